// cntr::convolution_timestep on device-resident herm_matrix data (libcntr
// cntr_convolution_impl.hpp:594-1803): C(n) = [A * B](n) for independent problems, each with its
// own C, A, Acc, B, Bcc in libcntr's layout (tv as ((t M + tau) s^2 + e)).  One launch covers up
// to NESSI_CONV_MAXP problems whose pointers travel in the kernel parameters, so a call needs no
// device allocation.
//   k_conv_ret   C^R(n, j)                 convolution_timestep_ret      (:741-899)
//   k_conv_tv    C^tv(n, tau)              convolution_timestep_tv       (:901-1073)
//   k_conv_les   C^<(j, n)                 convolution_timestep_les_*    (:1075-1580)
//   k_conv_mat   C^mat(tau)                convolution_matsubara         (:560-605)
// and k_conv_*_start for n < k, where the sums run to k with the hermitian continuations.  Work items
// of a problem are spread over blockIdx.x, problems over blockIdx.y.
//
// Bound of the steps n >= k: memory, the operands' triangles and tv rows once (A^R, B^R, A^<, A^tv,
// B^tv).  The lanes of a warp follow the index that is contiguous in memory and the sums are split
// over the warps of a CTA: k_conv_ret and k_conv_tv have a lane per (output index, column b), every
// warp takes each 8th term; k_conv_les has a CTA per JW consecutive rows j, a lane per term m, so that
// the right-hand blocks are loaded once for the JW rows and a column access A^<(j.., m) is a whole
// line.  Measured on a B200, 16 problems of size1 2, n 600, ntau 400 (ret / tv / les, us): a thread per
// output element, each summing alone, took 333 / 453 / 987; this form 81 / 90 / 228 (3.0 TB/s of
// operand bytes; one problem 137 us in all, before 1150).  The other sizes, 16 problems, n 200, ntau 100, all
// three, before and now: size1 1 466, 86; 3 825, 168; 4 865, 290; 5 1151, 601; 6 1338, 913; 7 1972, 1269; 8 3659,
// 2209; n 600, ntau 300: size1 5 5532, 5009 (16), size1 8 17947, 11300 (10 problems).
#pragma once
#include "device_common.cuh"

#define NESSI_CONV_MAXP 24  // 24 x 160 B of pointers keeps the parameters under 4 KB

struct ConvHM {
    double2 *ret, *les, *tv, *mat;
};
struct ConvProb {
    ConvHM C, A, Acc, B, Bcc;
};
struct ConvBatch {
    ConvProb p[NESSI_CONV_MAXP];
    int count, ntau, sig_a, sig_b, k;
    double h, beta;
};

__device__ __forceinline__ long ctri(long t) { return t * (t + 1) / 2; }

// element [a][b] of the s x s product X Y
template <int S>
__device__ __forceinline__ double2 emul(const double2 *X, const double2 *Y, int a, int b) {
    double2 t = cmk(0, 0);
#pragma unroll
    for (int c = 0; c < S; c++) t = cfma(X[a * S + c], Y[c * S + b], t);
    return t;
}
// element [a][b] of X Y^dagger
template <int S>
__device__ __forceinline__ double2 emul_ad(const double2 *X, const double2 *Y, int a, int b) {
    double2 t = cmk(0, 0);
#pragma unroll
    for (int c = 0; c < S; c++) t = cfma(X[a * S + c], cconj(Y[b * S + c]), t);
    return t;
}
// element [a][b] of X^dagger Y
template <int S>
__device__ __forceinline__ double2 emul_da(const double2 *X, const double2 *Y, int a, int b) {
    double2 t = cmk(0, 0);
#pragma unroll
    for (int c = 0; c < S; c++) t = cfma(cconj(X[c * S + a]), Y[c * S + b], t);
    return t;
}

// matsubara_integral_2 (conv_impl :410-540), element [a][d]: C(m) = c2 + sig c1 with
//   c1 = int_0^tau A(tau - x) B(beta - x) ..., c2 = int A(tau + x) B(x)  (rcorr near the ends)
// A and B are s x s blocks at A + t s^2 (t = 0..ntau).
template <int S>
__device__ double2 mat_int2(const double2 *A, const double2 *B, int m, int ntau, int k, double sg, int a, int d) {
    constexpr int s2 = S * S;
    double2 c1 = cmk(0, 0), c2 = cmk(0, 0);
    if (m == 0) {
    } else if (m < k) {
        for (int jj = 0; jj <= k; jj++)
            for (int l = 0; l <= k; l++)
                c1 = cfma(cmk(rcorr_w(k, m, l, jj), 0), emul<S>(A + jj * s2, B + (long)(ntau - l) * s2, a, d), c1);
    } else {
        for (int l = 0; l <= m; l++)
            c1 = cfma(cmk(greg_w(k, m, l), 0), emul<S>(A + (long)(m - l) * s2, B + (long)(ntau - l) * s2, a, d), c1);
    }
    const int r = ntau - m;
    if (r == 0) {
    } else if (r < k) {
        for (int l = 0; l <= k; l++)
            for (int jj = 0; jj <= k; jj++)
                c2 = cfma(cmk(rcorr_w(k, r, l, jj), 0), emul<S>(A + (long)(ntau - l) * s2, B + jj * s2, a, d), c2);
    } else {
        for (int l = 0; l <= r; l++)
            c2 = cfma(cmk(greg_w(k, r, l), 0), emul<S>(A + (long)(m + l) * s2, B + (long)l * s2, a, d), c2);
    }
    return cadd(c2, cscale(c1, sg));
}

// matsubara_integral_1 (conv_impl :86-224), element [a][d]: C(m) = c1 + sig c2 with
//   c1 = int_0^tau A(tau - x) B(x), c2 = int_tau^beta A(beta + tau - x) B(x)
template <int S>
__device__ double2 mat_int1(const double2 *A, const double2 *B, int m, int ntau, int k, double sg, int a, int d) {
    constexpr int s2 = S * S;
    double2 c1 = cmk(0, 0), c2 = cmk(0, 0);
    if (m >= k) {
        for (int j = 0; j <= m; j++)
            c1 = cfma(cmk(greg_w(k, m, j), 0), emul<S>(A + (long)(m - j) * s2, B + (long)j * s2, a, d), c1);
    } else if (m > 0) {
        for (int l = 0; l <= k; l++)
            for (int j = 0; j <= k; j++)
                c1 = cfma(cmk(rcorr_w(k, m, l, j), 0), emul<S>(A + (long)l * s2, B + (long)j * s2, a, d), c1);
    }
    const int r = ntau - m;
    if (r >= k) {
        for (int j = m; j <= ntau; j++)
            c2 = cfma(cmk(greg_w(k, r, ntau - j), 0), emul<S>(A + (long)(ntau - j + m) * s2, B + (long)j * s2, a, d), c2);
    } else if (r > 0) {
        for (int l = 0; l <= k; l++)
            for (int j = 0; j <= k; j++)
                c2 = cfma(cmk(rcorr_w(k, r, l, j), 0),
                          emul<S>(A + (long)(ntau - l) * s2, B + (long)(ntau - j) * s2, a, d), c2);
    }
    return cadd(c1, cscale(c2, sg));
}

// ---------------------------------------------------------------------------------------
// k_conv_ret_start: C^R(n,j) = h sum_m W(j,m) A^R(n,m) B^R(m,j) (convolution_timestep_ret, :741-899).
//   n < k:  m = 0..k with polynomial weights poly_integration(j, n, m) and the continuations
//           A^R(n,m) = -Acc^R(m,n)^dagger (m > n), B^R(m,j) = -Bcc^R(j,m)^dagger (m < j).
// ---------------------------------------------------------------------------------------
template <int S>
__global__ void k_conv_ret_start(ConvBatch cb, int n) {
    constexpr int s2 = S * S;
    const ConvProb &P = cb.p[blockIdx.y];
    const int k = cb.k;
    const double h = cb.h;
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < (long)(n + 1) * s2; e += (long)gridDim.x * blockDim.x) {
        const int j = (int)(e / s2), ab = (int)(e % s2), a = ab / S, b = ab % S;
        double2 acc = cmk(0, 0);
        {
            for (int m = 0; m <= k; m++) {
                double w = poly_int(k, j, n, m);
                double2 t = cmk(0, 0);
                for (int c = 0; c < S; c++) {
                    double2 av = n >= m ? P.A.ret[(ctri(n) + m) * s2 + a * S + c] : cconj(P.Acc.ret[(ctri(m) + n) * s2 + c * S + a]);
                    double2 bv = m >= j ? P.B.ret[(ctri(m) + j) * s2 + c * S + b] : cconj(P.Bcc.ret[(ctri(j) + m) * s2 + b * S + c]);
                    t = cfma(av, bv, t);
                }
                if (n < m) w = -w;
                if (m < j) w = -w;
                acc = cfma(cmk(w, 0), t, acc);
            }
        }
        P.C.ret[(ctri(n) + j) * s2 + ab] = cscale(acc, h);
    }
}

// ---------------------------------------------------------------------------------------
// k_conv_tv_start: C^tv(n,tau) = dtau matsubara_integral_2(A^tv(n,.), B^mat)(tau)
//                        + h sum_{j=0}^{max(n,k)} w(n,j) A'(n,j) B^tv(j,tau)   (:901-1073)
// with A'(n,j) = A^R(n,j) (j <= n) or -Acc^R(j,n)^dagger.
// ---------------------------------------------------------------------------------------
template <int S>
__global__ void k_conv_tv_start(ConvBatch cb, int n) {
    constexpr int s2 = S * S;
    const ConvProb &P = cb.p[blockIdx.y];
    const int k = cb.k, ntau = cb.ntau, M = ntau + 1, n1 = n > k ? n : k;
    const double h = cb.h, dtau = cb.beta / ntau;
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < (long)M * s2; e += (long)gridDim.x * blockDim.x) {
        const int m = (int)(e / s2), ab = (int)(e % s2), a = ab / S, b = ab % S;
        double2 acc = cscale(mat_int2<S>(P.A.tv + (long)n * M * s2, P.B.mat, m, ntau, k, (double)cb.sig_b, a, b), dtau);
        for (int j = 0; j <= n1; j++) {
            const double w = h * greg_w(k, n, j);
            const double2 *bt = P.B.tv + ((long)j * M + m) * s2;
            double2 t;
            if (j <= n) t = emul<S>(P.A.ret + (ctri(n) + j) * s2, bt, a, b);
            else t = cneg(emul_da<S>(P.Acc.ret + (ctri(j) + n) * s2, bt, a, b));
            acc = cfma(cmk(w, 0), t, acc);
        }
        P.C.tv[((long)n * M + m) * s2 + ab] = acc;
    }
}

// ---------------------------------------------------------------------------------------
// k_conv_les_start: C^<(j,n), j = 0..n (convolution_timestep_les, :1525-1580) as the sum of
//   tv*vt   sum_m w(ntau,m) A^tv(j,m) (-i dtau)(-sig_A) Bcc^tv(n,ntau-m)^dagger      (:1075-1242)
//   les*adv sum_m L(j,m) badv(m), L = A^< or -Acc^<(m,j)^dagger (m < j),
//           badv(m) = h w(n,m) Bcc^R(n,m)^dagger (m <= n) or -h w(n,m) B^R(m,n)       (:1244-1394)
//   ret*les sum_{m<=j} w(j,m) A^R(j,m) bl(m) [- sum_{m=j+1}^{k} w(j,m) Acc^R(m,j)^dagger bl(m), j < k],
//           bl(m) = h B^<(m,n) (m <= n) or -h Bcc^<(n,m)^dagger                        (:1396-1523)
// ---------------------------------------------------------------------------------------
template <int S>
__global__ void k_conv_les_start(ConvBatch cb, int n) {
    constexpr int s2 = S * S;
    const ConvProb &P = cb.p[blockIdx.y];
    const int k = cb.k, ntau = cb.ntau, M = ntau + 1, n1 = n > k ? n : k;
    const double h = cb.h, dtau = cb.beta / ntau;
    const double2 fvt = cmk(0.0, dtau * (double)cb.sig_a);  // (-i dtau)(-sig_A)
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < (long)(n + 1) * s2; e += (long)gridDim.x * blockDim.x) {
        const int j = (int)(e / s2), ab = (int)(e % s2), a = ab / S, b = ab % S;
        double2 acc = cmk(0, 0);
        // tv*vt
        for (int m = 0; m <= ntau; m++) {
            const double2 t = emul_ad<S>(P.A.tv + ((long)j * M + m) * s2, P.Bcc.tv + ((long)n * M + ntau - m) * s2, a, b);
            acc = cfma(cmul(fvt, cmk(greg_w(k, ntau, m), 0)), t, acc);
        }
        // les*adv
        for (int m = 0; m <= n1; m++) {
            const double w = h * greg_w(k, n, m);
            double2 t = cmk(0, 0);
            for (int c = 0; c < S; c++) {
                double2 lv = m >= j ? P.A.les[(ctri(m) + j) * s2 + a * S + c] : cneg(cconj(P.Acc.les[(ctri(j) + m) * s2 + c * S + a]));
                double2 bv = m <= n ? cscale(cconj(P.Bcc.ret[(ctri(n) + m) * s2 + b * S + c]), w)
                                    : cscale(P.B.ret[(ctri(m) + n) * s2 + c * S + b], -w);
                t = cfma(lv, bv, t);
            }
            acc = cadd(acc, t);
        }
        // ret*les
        for (int m = 0; m <= j; m++) {
            const double w = h * greg_w(k, j, m);
            acc = cfma(cmk(w, 0), emul<S>(P.A.ret + (ctri(j) + m) * s2, P.B.les + (ctri(n) + m) * s2, a, b), acc);
        }
        if (j < k)
            for (int m = j + 1; m <= k; m++) {
                const double w = h * greg_w(k, j, m);
                double2 t = cmk(0, 0);
                for (int c = 0; c < S; c++) {
                    double2 av = cconj(P.Acc.ret[(ctri(m) + j) * s2 + c * S + a]);
                    double2 bv = m <= n ? P.B.les[(ctri(n) + m) * s2 + c * S + b] : cneg(cconj(P.Bcc.les[(ctri(m) + n) * s2 + b * S + c]));
                    t = cfma(av, bv, t);
                }
                acc = cfma(cmk(-w, 0), t, acc);
            }
        P.C.les[(ctri(n) + j) * s2 + ab] = acc;
    }
}

// ---------------------------------------------------------------------------------------
// k_conv_ret, n >= k: C^R(n,j) = h sum_m W(j,m) A^R(n,m) B^R(m,j), m = j..n with W =
// gregory_weights(n-j, n-m) for m - j <= k, else 1 (m < n-k) or omega(n-m); for j > n-k also
// m = n-k..j-1 with B^R(m,j) = -Bcc^R(j,m)^dagger.  Lane = (j, b), 8 warps split m.
// ---------------------------------------------------------------------------------------
template <int S>
__global__ void __launch_bounds__(256) k_conv_ret(ConvBatch cb, int n) {
    constexpr int s2 = S * S;
    __shared__ double2 red[8 * 32 * S];
    const ConvProb &P = cb.p[blockIdx.y];
    const int k = cb.k, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int x = blockIdx.x * 32 + lane, j = x / S, b = x % S, j0 = (int)(blockIdx.x * 32) / S;
    const bool live = j <= n;
    double2 acc[S];
#pragma unroll
    for (int a = 0; a < S; a++) acc[a] = cmk(0, 0);
    const double2 *A = P.A.ret + ctri(n) * s2;
    const int mlo = min(j0, n - k);
#pragma unroll 4
    for (int m = mlo + warp; m <= n; m += 8) {
        if (!live || (m < j && m < n - k)) continue;
        double2 y[S];
        double w;
        if (m >= j) {
            const double2 *B = P.B.ret + (ctri(m) + j) * s2 + b;
#pragma unroll
            for (int c = 0; c < S; c++) y[c] = B[c * S];
            w = m - j <= k ? greg_w(k, n - j, n - m) : (m < n - k ? 1.0 : greg_omega(k, n - m));
        } else {
            const double2 *B = P.Bcc.ret + (ctri(j) + m) * s2 + b * S;
#pragma unroll
            for (int c = 0; c < S; c++) y[c] = cconj(B[c]);
            w = -greg_w(k, n - j, n - m);
        }
#pragma unroll
        for (int c = 0; c < S; c++) y[c] = cscale(y[c], w);
#pragma unroll
        for (int a = 0; a < S; a++)
#pragma unroll
            for (int c = 0; c < S; c++) acc[a] = cfma(A[(long)m * s2 + a * S + c], y[c], acc[a]);
    }
#pragma unroll
    for (int a = 0; a < S; a++) red[(a * 8 + warp) * 32 + lane] = acc[a];
    __syncthreads();
    for (int e = threadIdx.x; e < 32 * S; e += 256) {
        const int a = e / 32, l = e % 32, xx = blockIdx.x * 32 + l;
        double2 v = red[a * 256 + l];
#pragma unroll
        for (int w = 1; w < 8; w++) v = cadd(v, red[a * 256 + w * 32 + l]);
        if (xx / S <= n) P.C.ret[(ctri(n) + xx / S) * s2 + a * S + xx % S] = cscale(v, cb.h);
    }
}

// ---------------------------------------------------------------------------------------
// k_conv_tv, n >= k: C^tv(n,tau) = dtau matsubara_integral_2(A^tv(n,.), B^mat)(tau)
//                               + h sum_{j=0}^{n} w(n,j) A^R(n,j) B^tv(j,tau)   (:901-1073)
// Lane = (tau, b), 8 warps split j and the Matsubara sum (matsubara_integral_2 as in mat_int2).
// ---------------------------------------------------------------------------------------
// mat += w A B, column b of the block product (B points at column b)
template <int S>
__device__ __forceinline__ void cv_mat(double2 *mat, double w, const double2 *A, const double2 *B) {
#pragma unroll
    for (int c = 0; c < S; c++) {
        const double2 y = cscale(B[c * S], w);
#pragma unroll
        for (int a = 0; a < S; a++) mat[a] = cfma(A[a * S + c], y, mat[a]);
    }
}
template <int S>
__global__ void __launch_bounds__(256) k_conv_tv(ConvBatch cb, int n) {
    constexpr int s2 = S * S;
    __shared__ double2 red[8 * 32 * S];
    const ConvProb &P = cb.p[blockIdx.y];
    const int k = cb.k, ntau = cb.ntau, M = ntau + 1, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int x = blockIdx.x * 32 + lane, m = min(x / S, ntau), b = x % S, r = ntau - m;
    const double h = cb.h, dtau = cb.beta / ntau, sg = (double)cb.sig_b;
    double2 acc[S], mat[S];
#pragma unroll
    for (int a = 0; a < S; a++) acc[a] = mat[a] = cmk(0, 0);
    const double2 *A = P.A.ret + ctri(n) * s2, *B = P.B.tv + (long)m * s2 + b;
#pragma unroll 4
    for (int j = warp; j <= n; j += 8) {
        const double w = h * greg_w(k, n, j);
        double2 y[S];
#pragma unroll
        for (int c = 0; c < S; c++) y[c] = cscale(B[(long)j * M * s2 + c * S], w);
#pragma unroll
        for (int a = 0; a < S; a++)
#pragma unroll
            for (int c = 0; c < S; c++) acc[a] = cfma(A[(long)j * s2 + a * S + c], y[c], acc[a]);
    }
    const double2 *At = P.A.tv + (long)n * M * s2, *Bm = P.B.mat + b;
    for (int l = warp; l <= ntau; l += 8) {
        if (r >= k && l <= r) cv_mat<S>(mat, greg_w(k, r, l), At + (long)(m + l) * s2, Bm + (long)l * s2);
        if (m >= k && l <= m) cv_mat<S>(mat, sg * greg_w(k, m, l), At + (long)(m - l) * s2, Bm + (long)(ntau - l) * s2);
    }
    if ((r > 0 && r < k) || (m > 0 && m < k))
        for (int e = warp; e < (k + 1) * (k + 1); e += 8) {
            const int l = e / (k + 1), jj = e % (k + 1);
            if (r > 0 && r < k) cv_mat<S>(mat, rcorr_w(k, r, l, jj), At + (long)(ntau - l) * s2, Bm + (long)jj * s2);
            if (m > 0 && m < k) cv_mat<S>(mat, sg * rcorr_w(k, m, l, jj), At + (long)jj * s2, Bm + (long)(ntau - l) * s2);
        }
#pragma unroll
    for (int a = 0; a < S; a++)
        red[(a * 8 + warp) * 32 + lane] = cmk(fma(dtau, mat[a].x, acc[a].x), fma(dtau, mat[a].y, acc[a].y));
    __syncthreads();
    for (int e = threadIdx.x; e < 32 * S; e += 256) {
        const int a = e / 32, l = e % 32, xx = blockIdx.x * 32 + l;
        double2 v = red[a * 256 + l];
#pragma unroll
        for (int w = 1; w < 8; w++) v = cadd(v, red[a * 256 + w * 32 + l]);
        if (xx / S <= ntau) P.C.tv[((long)n * M + xx / S) * s2 + a * S + xx % S] = v;
    }
}

// ---------------------------------------------------------------------------------------
// k_conv_les, n >= k: C^<(j,n), j = 0..n, as the sum of
//   tv*vt   sum_m w(ntau,m) A^tv(j,m) (-i dtau)(-sig_A) Bcc^tv(n,ntau-m)^dagger      (:1075-1242)
//   les*adv sum_m L(j,m) badv(m), L = A^< or -Acc^<(m,j)^dagger (m < j),
//           badv(m) = h w(n,m) Bcc^R(n,m)^dagger                                      (:1244-1394)
//   ret*les sum_{m<=j} w(j,m) A^R(j,m) h B^<(m,n) [- sum_{m=j+1}^{k} w(j,m) Acc^R(m,j)^dagger h B^<(m,n),
//           j < k]                                                                    (:1396-1523)
// A CTA of 4 warps takes JW rows j; lanes split m; CB columns b of the s x s blocks at a time.
// ---------------------------------------------------------------------------------------
template <int S> struct CvCfg {
    static constexpr int JW = S == 1 ? 8 : (S == 2 ? 4 : (S == 3 ? 2 : 1));
    static constexpr int CB = S <= 4 ? S : 2;
};
// acc += w L' R, L' = L or (tr) L^dagger, an s x s block; R s x CB
template <int S, int CB>
__device__ __forceinline__ void cv_fold(double2 (*acc)[CB], const double2 *L, bool tr, double w, const double2 (*R)[CB]) {
#pragma unroll
    for (int a = 0; a < S; a++)
#pragma unroll
        for (int c = 0; c < S; c++) {
            double2 l = L[tr ? c * S + a : a * S + c];
            l = cmk(l.x * w, l.y * (tr ? -w : w));
#pragma unroll
            for (int e = 0; e < CB; e++) acc[a][e] = cfma(l, R[c][e], acc[a][e]);
        }
}
template <int S>
__global__ void __launch_bounds__(128) k_conv_les(ConvBatch cb, int n) {
    constexpr int s2 = S * S, JW = CvCfg<S>::JW, CB = CvCfg<S>::CB, NE = JW * S * CB;
    __shared__ double2 red[NE * 4];
    const ConvProb &P = cb.p[blockIdx.y];
    const int k = cb.k, ntau = cb.ntau, M = ntau + 1, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double h = cb.h, dtau = cb.beta / ntau, fvt = dtau * (double)cb.sig_a;  // (-i dtau)(-sig_A) = i fvt
    const int j0 = blockIdx.x * JW;
    for (int c0 = 0; c0 < S; c0 += CB) {
        double2 acc[JW][S][CB];
#pragma unroll
        for (int q = 0; q < JW; q++)
#pragma unroll
            for (int a = 0; a < S; a++)
#pragma unroll
                for (int e = 0; e < CB; e++) acc[q][a][e] = cmk(0, 0);
        double2 R[S][CB];
        // tv*vt
        for (int m = tid; m <= ntau; m += 128) {
            const double w = fvt * greg_w(k, ntau, m);
            const double2 *B = P.Bcc.tv + ((long)n * M + ntau - m) * s2;
#pragma unroll
            for (int c = 0; c < S; c++)
#pragma unroll
                for (int e = 0; e < CB; e++) {  // i w B^dagger
                    const double2 v = c0 + e < S ? B[(c0 + e) * S + c] : cmk(0, 0);
                    R[c][e] = cmk(w * v.y, w * v.x);
                }
#pragma unroll
            for (int q = 0; q < JW; q++)
                cv_fold<S, CB>(acc[q], P.A.tv + ((long)min(j0 + q, n) * M + m) * s2, false, 1.0, R);
        }
        // les*adv
        for (int m = tid; m <= n; m += 128) {
            const double w = h * greg_w(k, n, m);
            const double2 *B = P.Bcc.ret + (ctri(n) + m) * s2;
#pragma unroll
            for (int c = 0; c < S; c++)
#pragma unroll
                for (int e = 0; e < CB; e++) R[c][e] = c0 + e < S ? cscale(cconj(B[(c0 + e) * S + c]), w) : cmk(0, 0);
#pragma unroll
            for (int q = 0; q < JW; q++) {
                const int j = min(j0 + q, n);
                const bool up = m >= j;
                const double2 *L = up ? P.A.les + (ctri(m) + j) * s2 : P.Acc.les + (ctri(j) + m) * s2;
                cv_fold<S, CB>(acc[q], L, !up, up ? 1.0 : -1.0, R);
            }
        }
        // ret*les (rows j < k: to k, with the continuation of A)
        const int jmax = min(j0 + JW - 1, n), mhi = max(jmax, j0 < k ? k : 0);
        for (int m = tid; m <= mhi; m += 128) {
            const double2 *B = P.B.les + (ctri(n) + m) * s2;
#pragma unroll
            for (int c = 0; c < S; c++)
#pragma unroll
                for (int e = 0; e < CB; e++) R[c][e] = c0 + e < S ? cscale(B[c * S + c0 + e], h) : cmk(0, 0);
#pragma unroll
            for (int q = 0; q < JW; q++) {
                const int j = min(j0 + q, n);
                if (m > j && (j >= k || m > k)) continue;
                const bool low = m <= j;
                const double w = low ? greg_w(k, j, m) : -greg_w(k, j, m);
                const double2 *L = low ? P.A.ret + (ctri(j) + m) * s2 : P.Acc.ret + (ctri(m) + j) * s2;
                cv_fold<S, CB>(acc[q], L, !low, w, R);
            }
        }
        // sum over the lanes, then over the warps
#pragma unroll
        for (int q = 0; q < JW; q++)
#pragma unroll
            for (int a = 0; a < S; a++)
#pragma unroll
                for (int e = 0; e < CB; e++) {
                    double2 v = acc[q][a][e];
#pragma unroll
                    for (int off = 16; off > 0; off >>= 1) {
                        v.x += __shfl_xor_sync(0xffffffffu, v.x, off);
                        v.y += __shfl_xor_sync(0xffffffffu, v.y, off);
                    }
                    if (lane == 0) red[((q * S + a) * CB + e) * 4 + warp] = v;
                }
        __syncthreads();
        for (int x = tid; x < NE; x += 128) {
            const int q = x / (S * CB), a = (x / CB) % S, e = x % CB;
            const double2 v = cadd(cadd(red[x * 4], red[x * 4 + 1]), cadd(red[x * 4 + 2], red[x * 4 + 3]));
            if (j0 + q <= n && c0 + e < S) P.C.les[(ctri(n) + j0 + q) * s2 + a * S + c0 + e] = v;
        }
        __syncthreads();
    }
}

// k_conv_mat: C^mat(tau) = dtau matsubara_integral_1(A^mat, B^mat)(tau), sig of A (:560-582)
template <int S>
__global__ void k_conv_mat(ConvBatch cb) {
    constexpr int s2 = S * S;
    const ConvProb &P = cb.p[blockIdx.y];
    const int k = cb.k, ntau = cb.ntau, M = ntau + 1;
    const double dtau = cb.beta / ntau;
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < (long)M * s2; e += (long)gridDim.x * blockDim.x) {
        const int m = (int)(e / s2), ab = (int)(e % s2), a = ab / S, b = ab % S;
        P.C.mat[(long)m * s2 + ab] = cscale(mat_int1<S>(P.A.mat, P.B.mat, m, ntau, k, (double)cb.sig_a, a, b), dtau);
    }
}
