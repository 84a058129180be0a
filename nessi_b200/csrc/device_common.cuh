// Device helpers shared by the Kadanoff-Baym kernels: complex arithmetic on double2,
// the integration tables in constant memory, Gregory weight lookup and a CTA-wide
// dense complex solver for the (k*s) x (k*s) start blocks.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "cntr_tables.inc"

#define NESSI_MAXS 8        // largest orbital size with a compiled kernel
#define NESSI_K1MAX (CNTR_KMAX + 1)
#define NESSI_K2MAX (2 * NESSI_K1MAX)

// ---- complex arithmetic (double2 = re, im) -----------------------------------------
__host__ __device__ __forceinline__ double2 cmk(double r, double i) { return make_double2(r, i); }
__host__ __device__ __forceinline__ double2 cadd(double2 a, double2 b) { return cmk(a.x + b.x, a.y + b.y); }
__host__ __device__ __forceinline__ double2 csub(double2 a, double2 b) { return cmk(a.x - b.x, a.y - b.y); }
__host__ __device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return cmk(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// c + a*b
__host__ __device__ __forceinline__ double2 cfma(double2 a, double2 b, double2 c) {
    return cmk(fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y)));
}
__host__ __device__ __forceinline__ double2 cscale(double2 a, double s) { return cmk(a.x * s, a.y * s); }
__host__ __device__ __forceinline__ double2 cconj(double2 a) { return cmk(a.x, -a.y); }
__host__ __device__ __forceinline__ double2 cneg(double2 a) { return cmk(-a.x, -a.y); }
__host__ __device__ __forceinline__ double2 cdiv(double2 a, double2 b) {
    // Smith's algorithm
    if (fabs(b.x) >= fabs(b.y)) {
        double r = b.y / b.x, d = b.x + b.y * r;
        return cmk((a.x + a.y * r) / d, (a.y - a.x * r) / d);
    } else {
        double r = b.x / b.y, d = b.x * r + b.y;
        return cmk((a.x * r + a.y) / d, (a.y * r - a.x) / d);
    }
}
__host__ __device__ __forceinline__ double cabs2(double2 a) { return a.x * a.x + a.y * a.y; }

// ---- overlapped launches (programmatic stream serialization) --------------------------------
// A kernel launched with launch_chained may start while its predecessor in the stream still runs.  It
// waits (pdl_wait) before it reads or writes anything another kernel touches; since every kernel of a
// chain does, "the predecessor has finished" implies that all earlier ones have.  What the kernels of a
// chain write is read by ordinary or cp.async loads only: the read-only path (__ldg, or a const
// __restrict__ pointer) is for data that no kernel writes while the reader is resident, and pdl_wait does
// not order it.  pdl_trigger lets the
// successor's CTAs take free SM resources once all CTAs of this kernel have started; long streaming
// kernels leave it out, so that waiting CTAs do not sit beside them.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_entry() {
    pdl_trigger();
    pdl_wait();
}

// ---- integration tables (one order k per launch; indexed [k]) ----------------------
struct IntegTables {
    double greg[NESSI_K1MAX][NESSI_K2MAX * NESSI_K2MAX];
    double omega[NESSI_K1MAX][NESSI_K1MAX];
    double poly_int[NESSI_K1MAX][NESSI_K1MAX * NESSI_K1MAX * NESSI_K1MAX];
    double poly_diff[NESSI_K1MAX][NESSI_K1MAX * NESSI_K1MAX];
    double poly_interp[NESSI_K1MAX][NESSI_K1MAX * NESSI_K1MAX];
    double bd[NESSI_K1MAX][NESSI_K1MAX + 1];
    double rcorr[NESSI_K1MAX][(NESSI_K1MAX - 2) * NESSI_K1MAX * NESSI_K1MAX];
};
__constant__ IntegTables c_tab;  // single translation unit (nessi_gpu.cu)

// Integrator::gregory_weights(n, j) (integration.hpp:382-390) for order k.
__device__ __forceinline__ double greg_w(int k, int n, int j) {
    const int k1 = k + 1, k2 = 2 * k1;
    if (n >= k2) {
        if (j > k && j < n - k) return 1.0;
        if (j < k1) return c_tab.omega[k][j];
        return c_tab.omega[k][n - j];
    }
    return c_tab.greg[k][n * NESSI_K2MAX + j];
}
__device__ __forceinline__ double greg_omega(int k, int j) { return c_tab.omega[k][j]; }
__device__ __forceinline__ double poly_diff(int k, int i, int l) { return c_tab.poly_diff[k][i * NESSI_K1MAX + l]; }
__device__ __forceinline__ double poly_int(int k, int i, int j, int l) {
    return c_tab.poly_int[k][(i * NESSI_K1MAX + j) * NESSI_K1MAX + l];
}
__device__ __forceinline__ double bd_w(int k, int l) { return c_tab.bd[k][l]; }
__device__ __forceinline__ double rcorr_w(int k, int m, int j, int l) {
    if (k < 2) return 0.0;
    return c_tab.rcorr[k][((m - 1) * NESSI_K1MAX + j) * NESSI_K1MAX + l];
}

// ---- dense solve A X = B (n x n, nrhs columns), partial pivoting, by the whole CTA -------------
// A (n x n, row-major, lda = n) and B (n x nrhs, row-major) live in shared memory and
// are overwritten; on return B holds X.  Every thread of the CTA must call it.
// Returns nonzero in *status (shared) if a zero pivot was met.
// Bound: the chain of n columns; per column the pivot search (the first warp), one division per
// row, and the update of the rest, then as many steps of a column-wise back substitution.
__device__ inline void grp_solve(double2 *A, double2 *B, int n, int nrhs, int *s_piv, int *status) {
    const int tid = threadIdx.x, nth = blockDim.x;
    for (int c = 0; c < n; c++) {
        if (tid < 32) {
            int p = c;
            double best = -1.0;
            for (int i = c + tid; i < n; i += 32) {
                const double a = cabs2(A[i * n + c]);
                if (a > best) { best = a; p = i; }
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                const double ob = __shfl_xor_sync(0xffffffffu, best, off);
                const int op = __shfl_xor_sync(0xffffffffu, p, off);
                if (ob > best || (ob == best && op < p)) { best = ob; p = op; }
            }
            if (tid == 0) {
                *s_piv = p;
                if (best == 0.0) *status = 1;
            }
        }
        __syncthreads();
        const int p = *s_piv;
        if (p != c)
            for (int j = tid; j < n + nrhs; j += nth) {
                double2 *u = j < n ? A + c * n + j : B + c * nrhs + j - n, *v = j < n ? A + p * n + j : B + p * nrhs + j - n;
                const double2 t = *u;
                *u = *v;
                *v = t;
            }
        __syncthreads();
        double2 piv = A[c * n + c];
        if (piv.x == 0.0 && piv.y == 0.0) piv = cmk(1.0, 0.0);  // status already flagged
        for (int i = c + 1 + tid; i < n; i += nth) A[i * n + c] = cdiv(A[i * n + c], piv);
        __syncthreads();
        // eliminate rows below c
        const int w = n - c - 1 + nrhs;  // columns c+1..n-1 and rhs
        for (int idx = tid; idx < (n - c - 1) * w; idx += nth) {
            const int i = c + 1 + idx / w, j = idx % w;
            const double2 f = A[i * n + c];
            double2 *u = j < n - c - 1 ? A + i * n + c + 1 + j : B + i * nrhs + j - (n - c - 1);
            const double2 *v = j < n - c - 1 ? A + c * n + c + 1 + j : B + c * nrhs + j - (n - c - 1);
            *u = csub(*u, cmul(f, *v));
        }
        __syncthreads();
    }
    // back substitution, column by column
    for (int i = n - 1; i >= 0; i--) {
        double2 d = A[i * n + i];
        if (d.x == 0.0 && d.y == 0.0) d = cmk(1.0, 0.0);
        for (int j = tid; j < nrhs; j += nth) B[i * nrhs + j] = cdiv(B[i * nrhs + j], d);
        __syncthreads();
        for (int idx = tid; idx < i * nrhs; idx += nth) {
            const int r = idx / nrhs, j = idx % nrhs;
            B[idx] = csub(B[idx], cmul(A[r * n + i], B[i * nrhs + j]));
        }
        __syncthreads();
    }
}

// The same for n <= 32 by one warp, a row per lane: no rows are exchanged (a lane remembers the column
// its row is the pivot of), the pivot comes from one 32-bit maximum over the leading words of the
// candidates' larger component, and every lane has the reciprocal of its candidate ready by then.
// Bound: the chain of n columns, about 500 cycles each, and 200 per row of the back substitution.
__device__ inline void warp_solve(double2 *A, double2 *B, int n, int nrhs, int *status) {
    const unsigned all = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    double2 *Ar = A + lane * n, *Br = B + lane * nrhs, rp = cmk(1.0, 0.0);
    int ord = lane < n ? -1 : n;  // the column this row is the pivot of
    for (int c = 0; c < n; c++) {
        const bool cand = ord < 0;
        const double2 v = cand ? Ar[c] : cmk(0, 0);
        const double m = cabs2(v), im = 1.0 / m;
        const unsigned key = cand ? 1u + (unsigned)__double2hiint(fmax(fabs(v.x), fabs(v.y))) : 0u;
        const unsigned best = __reduce_max_sync(all, key);
        const int p = __ffs(__ballot_sync(all, key == best)) - 1;
        double2 r = cmk(v.x * im, -v.y * im);
        if (lane == p) {
            if (!(m > 1e-290 && m < 1e290)) {  // the square left the range of a double
                if (v.x == 0.0 && v.y == 0.0) *status = 1;
                r = v.x == 0.0 && v.y == 0.0 ? cmk(1.0, 0.0) : cdiv(cmk(1.0, 0.0), v);
            }
            ord = c;
            rp = r;
        }
        r = cmk(__shfl_sync(all, r.x, p), __shfl_sync(all, r.y, p));
        if (ord < 0) {
            const double2 f = cmul(v, r);
            const double2 *Ap = A + p * n, *Bp = B + p * nrhs;
            for (int j = c + 1; j < n; j++) Ar[j] = csub(Ar[j], cmul(f, Ap[j]));
            for (int j = 0; j < nrhs; j++) Br[j] = csub(Br[j], cmul(f, Bp[j]));
        }
        __syncwarp();
    }
    for (int i = n - 1; i >= 0; i--) {
        const int p = __ffs(__ballot_sync(all, ord == i)) - 1;
        if (lane == p)
            for (int j = 0; j < nrhs; j++) Br[j] = cmul(Br[j], rp);
        __syncwarp();
        if (ord < i) {
            const double2 f = Ar[i], *Bp = B + p * nrhs;
            for (int j = 0; j < nrhs; j++) Br[j] = csub(Br[j], cmul(f, Bp[j]));
        }
        __syncwarp();
    }
    for (int j = 0; j < nrhs; j++) {  // rows back into the order of the unknowns
        const double2 x = lane < n ? Br[j] : cmk(0, 0);
        __syncwarp();
        if (lane < n) B[ord * nrhs + j] = x;
        __syncwarp();
    }
}

// Small systems by the CTA's first warp, the others by the whole CTA.  Start rows of a step in us, warp / CTA:
// size1 1 (5 unknowns, one problem) 9 / 13, size1 2 (10 unknowns, 32 problems) 16 / 22, size1 4 (20 unknowns
// and 4 right-hand sides, 32 problems) 32 / 38.  Above, a row per lane leaves too much to one warp.
__device__ inline void cta_solve(double2 *A, double2 *B, int n, int nrhs, int *s_piv, int *status) {
    if (n <= 32 && n * (n + nrhs) <= 700) {
        if (threadIdx.x < 32) warp_solve(A, B, n, nrhs, status);
        __syncthreads();
    } else {
        grp_solve(A, B, n, nrhs, s_piv, status);
    }
}

// Invert an s x s complex matrix held by one thread (Gauss-Jordan, partial pivoting).
template <int S>
__device__ inline int small_inverse(const double2 *M, double2 *Minv) {
    double2 a[S][2 * S];
    for (int i = 0; i < S; i++)
        for (int j = 0; j < S; j++) {
            a[i][j] = M[i * S + j];
            a[i][S + j] = cmk(i == j ? 1.0 : 0.0, 0.0);
        }
    int bad = 0;
    for (int c = 0; c < S; c++) {
        int p = c;
        double best = cabs2(a[c][c]);
        for (int i = c + 1; i < S; i++)
            if (cabs2(a[i][c]) > best) { best = cabs2(a[i][c]); p = i; }
        if (best == 0.0) { bad = 1; continue; }
        if (p != c)
            for (int j = 0; j < 2 * S; j++) { double2 t = a[c][j]; a[c][j] = a[p][j]; a[p][j] = t; }
        double2 inv = cdiv(cmk(1, 0), a[c][c]);
        for (int j = 0; j < 2 * S; j++) a[c][j] = cmul(a[c][j], inv);
        for (int i = 0; i < S; i++) {
            if (i == c) continue;
            double2 f = a[i][c];
            for (int j = 0; j < 2 * S; j++) a[i][j] = csub(a[i][j], cmul(f, a[c][j]));
        }
    }
    for (int i = 0; i < S; i++)
        for (int j = 0; j < S; j++) Minv[i * S + j] = a[i][S + j];
    return bad;
}
