// Batched Dyson time step (libcntr cntr_dyson_impl.hpp:1618-1648) for many problems
// ("k-points") sharing one self-energy Sigma.  Every problem keeps libcntr's herm_matrix
// layout in device memory (cntr_herm_matrix_impl.hpp:457-477).
//
// One time step n > k runs as
//   k_prep           s x s inverses of the step matrices (dyson_impl :179-213, :693-706, :983-1011),
//                    history coefficients for tv, dense copies of Sigma^< and Sigma^tv
//   ret recursion    G^R(n, 0..n): k-block start + Volterra recursion in t'   (:80-222)
//   k_tv_ring        G^tv(n, 0..ntau): (k_tv_mixed with the FP32 copy of the history)
//                    history stream + Matsubara integral + solve (:651-741)
//   k_les_operands_t right-hand operands of the Sigma-shared products
//   k_zgemm products     tv*vt + les*adv convolutions for all problems at once (conv_impl :1075-1394)
//   les recursion    G^<(0..n, n): k-block start + Volterra recursion in t (:893-1056)
// The recursions are in kernels_recursion.cuh.
#pragma once
#include "device_common.cuh"
#include "kernels_gemm.cuh"

struct ProbDev {
    double2 *gret, *gles, *gtv, *gmat;  // this problem's G (libcntr layout)
    const double2 *qret, *qles, *qtv;   // VIE2: the source term Q (tv in plane layout); else null
    const double2 *H;                   // (nt+2) s^2 blocks, H(-1) first
    double2 *minv_ret, *minv_les;       // (nt+1) s^2: inverses of the ret / les+tv step matrices
    float2 *gtv32;                      // mixed precision: FP32 copy of G^tv (plane layout) or null
    double mu;
    int nt;
    int col;                            // column of this problem in the group's GEMM operands
    int pad;
};

struct GroupDev {
    const double2 *sret, *sles, *stv, *smat;  // Sigma, or F of a VIE2 group (libcntr layout, shared)
    const double2 *rret;  // triangle of the retarded recursion: Sigma^R, or Fcc^R for VIE2
    const double2 *lcc;   // lesser triangle for t' < t of the les*adv operand: Sigma^<, or Fcc^<
    double2 *Ldense;   // ((ntmax+1)s) x ((ntmax+1)s) row-major: Sigma^<(j,m), full (anti-hermitian)
    double2 *Tdense;   // ((ntmax+1)s) x ((ntau+1)s) row-major: Sigma^tv(j,m) reordered (s>1)
    double2 *tvcoef;   // (ntmax+1) s^2: coefficients of the tv history sum at the current step
    double2 *badv, *btv, *gles;  // GEMM operands / result, leading dimension ldc
    double2 *Kmat;     // ((ntau+1)s) x ((ntau+1)s) row-major: Matsubara operator of the step
    double2 *Gmat_all; // ((ntau+1)s) x ldc: every problem's G^mat as columns
    double2 *Cmat;     // ((ntau+1)s) x ldc: Matsubara part of the tv right-hand side
    const double2 *fccmat;  // Fcc^mat of a VIE2 group (steepest-descent vie2_mat), or null
    double2 *vy, *vacc;     // ((ntmax+1)s) x ldc: solved rows and far sums of the blocked recursion
    double2 *vst;           // ((k+1)s) x ldc: its start rows
    const ProbDev *probs;   // the group's problems, nt descending
    int ntmax, ntau, s, sig, k;
    int ldc;           // >= nprob * s
    double h, beta;
    double conv_sign;  // sign of the convolutions on the right-hand side: 1 (Dyson), -1 (VIE2)
};

#define NESSI_GSEL 64  // groups per launch
// The groups of a launch (blockIdx.y or .z): index into the batch's group table, active problems
struct GroupSel {
    int ng;
    int gid[NESSI_GSEL], nact[NESSI_GSEL];
};
// First time indices a step has to prepare, per group of a GroupSel: step matrices of the lesser / tv
// and retarded equations, dense rows and columns of Sigma
struct PrepSel {
    int les_lo[NESSI_GSEL], ret_lo[NESSI_GSEL], d_lo[NESSI_GSEL];
};

__device__ __forceinline__ long tri(long t) { return t * (t + 1) / 2; }

// ---------------------------------------------------------------------------------------
// prep_problem: Minv_les[n] (= tv step matrix for n > k), Minv_ret[j] for j in [r0, r1]
//   tv/les:  mm = i/h bd0 + mu - H(n) - h w0 Sigma^R(n,n)        (dyson_impl :693-699, :983-1004)
//   ret:     mm = i/h bd0 + mu - H(j)^dagger - h w0 Sigma^R(j,j) (dyson_impl :188-199)
// ---------------------------------------------------------------------------------------
// VIE2 ([1 + F] G = Q, cntr_vie2_impl.hpp:60-140, 645-725, 847-990): the step matrices are
//   tv/les:  mm = 1 + h w0 F^R(j,j);   ret: mm = 1 + h w0 Fcc^R(j,j)
template <int S, bool VIE>
__device__ __forceinline__ void prep_problem(const GroupDev &g, const ProbDev &p, int n, int les_lo, int r0) {
    const int k = g.k, s2 = S * S, r1 = n - k - 1;
    const double h = g.h;
    const double2 ibd0 = cmk(0.0, bd_w(k, 0) / h);
    const double w0 = h * greg_omega(k, 0);
    // rows: les indices les_lo..n then ret indices r0..r1
    int nles = n - les_lo + 1;
    int nret = r1 >= r0 ? r1 - r0 + 1 : 0;
    for (int t = threadIdx.x; t < nles + nret; t += blockDim.x) {
        bool is_ret = t >= nles;
        int j = is_ret ? r0 + (t - nles) : les_lo + t;
        if (j > p.nt) continue;
        double2 M[S * S];
        if (VIE) {
            const double2 *Fjj = (is_ret ? g.rret : g.sret) + (tri(j) + j) * s2;
            for (int e = 0; e < s2; e++) M[e] = cadd(cscale(Fjj[e], w0), cmk(e / S == e % S ? 1.0 : 0.0, 0.0));
        } else {
            const double2 *Hj = p.H + (long)(j + 1) * s2;
            const double2 *Sjj = g.sret + (tri(j) + j) * s2;
            for (int a = 0; a < S; a++)
                for (int b = 0; b < S; b++) {
                    double2 hv = is_ret ? cconj(Hj[b * S + a]) : Hj[a * S + b];
                    double2 v = csub(cscale(Sjj[a * S + b], -w0), hv);
                    if (a == b) v = cadd(v, cadd(ibd0, cmk(p.mu, 0.0)));
                    M[a * S + b] = v;
                }
        }
        double2 *dst = (is_ret ? p.minv_ret : p.minv_les) + (long)j * s2;
        small_inverse<S>(M, dst);
    }
}

// ---------------------------------------------------------------------------------------
// prep_group: tv coefficients a_j = h w(n,j) Sigma^R(n,j) - [n-k-1<=j<n] (i/h) bd(n-j) 1
// (conv_impl :942-972 with the BDF terms of dyson_impl :681-692 folded in), and the dense
// copies of Sigma^< (rows/columns d_lo..n) and Sigma^tv (rows d_lo..n).
// ---------------------------------------------------------------------------------------
// VIE2: a_j = -h w(n,j) F^R(n,j) (conv_tv with A = F, moved to the right-hand side).
template <int S, bool VIE>
__device__ __forceinline__ void prep_group(const GroupDev &g, int n, int d_lo, int blk, int nblk) {
    const int k = g.k, s2 = S * S;
    const double h = g.h;
    const long tid = blk * (long)blockDim.x + threadIdx.x;
    const long nth = (long)nblk * blockDim.x;
    // tv coefficients, j = 0..n-1
    for (long e = tid; e < (long)n * s2; e += nth) {
        int j = (int)(e / s2), ab = (int)(e % s2), a = ab / S, b = ab % S;
        double2 v = cscale(g.sret[(tri(n) + j) * s2 + ab], (VIE ? -h : h) * greg_w(k, n, j));
        if (!VIE && j >= n - k - 1 && a == b) v = csub(v, cmk(0.0, bd_w(k, n - j) / h));
        g.tvcoef[(long)j * s2 + ab] = v;
    }
    // dense Sigma^<: for every t in [d_lo, n]: column t (rows 0..t) and row t (cols 0..t-1)
    const long ldL = (long)(g.ntmax + 1) * S;
    for (int t = d_lo; t <= n; t++) {
        for (long e = tid; e < (long)(t + 1) * s2; e += nth) {
            int j = (int)(e / s2), ab = (int)(e % s2), a = ab / S, b = ab % S;
            // L(j,t) = Sigma^<(j,t), j <= t
            double2 v = g.sles[(tri(t) + j) * s2 + ab];
            g.Ldense[((long)j * S + a) * ldL + (long)t * S + b] = v;
            // L(t,j) = -Sigma^<(j,t)^dagger (-Fcc^<(j,t)^dagger for VIE2), j < t  [element (b,a)]
            if (j < t) g.Ldense[((long)t * S + b) * ldL + (long)j * S + a] = cneg(cconj(g.lcc[(tri(t) + j) * s2 + ab]));
        }
    }
    if (S > 1) {
        const long ldT = (long)(g.ntau + 1) * S;
        for (int t = d_lo; t <= n; t++)
            for (long e = tid; e < (long)(g.ntau + 1) * s2; e += nth) {
                int m = (int)(e / s2), ab = (int)(e % s2), a = ab / S, b = ab % S;
                g.Tdense[((long)t * S + a) * ldT + (long)m * S + b] =
                    g.stv[((long)t * (g.ntau + 1) + m) * s2 + ab];
            }
    }
}

// k_prep: the step matrices and the dense operands of a step, one launch: blocks 0..np-1 the step
// matrices (a problem each), the rest prep_group.  Grid (np + prep_group blocks, groups).
template <int S, bool VIE>
__global__ void __launch_bounds__(256) k_prep(const GroupDev *__restrict__ gt, GroupSel sel, PrepSel ps, int n, int np) {
    pdl_entry();
    const int y = blockIdx.y, x = blockIdx.x;
    const GroupDev &g = gt[sel.gid[y]];
    if (x >= np) prep_group<S, VIE>(g, n, ps.d_lo[y], x - np, (int)gridDim.x - np);
    else if (x < sel.nact[y]) prep_problem<S, VIE>(g, g.probs[x], n, ps.les_lo[y], ps.ret_lo[y]);
}

// ---------------------------------------------------------------------------------------
// Start blocks: the k x k block systems of dyson_timestep_ret (:112-157) and
// dyson_timestep_les (:926-982), solved by the whole CTA in shared memory.
// ---------------------------------------------------------------------------------------
// A thread per matrix element: its terms are loaded independently, so the assembly costs a few memory
// latencies, not one per term.
// ret: unknowns X_q = G(n, n-q-1); equations sum_q X_q mm(p,q) = qq(p)  (left solve), solved as the
// right solve of the block-wise adjoints: A[(p,a),(q,b)] = conj(mm(p,q)[b][a]), R[(p,a),c] = conj(qq(p)[c][a]).
// Dyson, j = p+1, l = q+1, stemp(l) = Sigma(n-l, n-j) (l <= j) or -Sigma(n-j, n-l)^dagger:
//   mm(p,q) = (i/h) P(j,l) 1 + delta_lj (mu - H(n-j)) - h w(j,l) stemp(l)
//   qq(p) = -(i/h) P(j,0) G(n,n) + h w(j,0) G(n,n) stemp(0),  G(n,n) = -i 1
// VIE2 (vie2_timestep_ret, cntr_vie2_impl.hpp:60-140, called with F and Fcc swapped), G(n,n) = Q(n,n) set,
// F'(t,t') = Fcc^R(t,t') for t >= t' and -F^R(t',t)^dagger otherwise:
//   mm(p,q) = 1 delta_pq + h w(j,l) F'(n-l, n-j),  qq(p) = Q(n, n-j) - h w(j,0) G(n,n) F'(n, n-j)
template <int S, bool VIE>
__device__ void ret_start_block(const GroupDev &g, const ProbDev &p, int n, double2 *smem) {
    const int k = g.k, s2 = S * S, KS = k * S;
    const double h = g.h;
    double2 *A = smem;           // (KS x KS)
    double2 *R = A + KS * KS;    // (KS x S)
    int *ipiv = (int *)(R + KS * S);
    int *status = ipiv + 1;
    double2 *grow = p.gret + tri(n) * s2;  // G(n, .)
    if (threadIdx.x == 0) *status = 0;
    for (int e = threadIdx.x; e < KS * (KS + S); e += blockDim.x) {
        const int r = e / (KS + S), c = e % (KS + S), j = r / S + 1, b = r % S;
        if (c < KS) {  // element mm(j-1, l-1)[a][b]
            const int l = c / S + 1, a = c % S;
            double w = h * greg_w(k, j, l);
            double2 st;
            if (l <= j) {
                st = g.rret[(tri(n - l) + n - j) * s2 + a * S + b];
            } else {
                st = cconj(g.sret[(tri(n - j) + n - l) * s2 + b * S + a]);
                w = -w;
            }
            double2 v = cmk(0, 0);
            if (VIE) {
                if (l == j && a == b) v = cmk(1.0, 0.0);
                v = cadd(v, cscale(st, w));
            } else {
                if (a == b) v = cmk(0.0, poly_diff(k, j, l) / h);
                if (l == j) {
                    double2 u = cneg(p.H[(long)(n - j + 1) * s2 + a * S + b]);
                    if (a == b) u = cadd(u, cmk(p.mu, 0.0));
                    v = cadd(v, u);
                }
                v = csub(v, cscale(st, w));
            }
            A[r * KS + c] = cconj(v);
        } else {  // element qq(j-1)[a][b]
            const int a = c - KS;
            const double w = h * greg_w(k, j, 0);
            const double2 *fr = g.rret + (tri(n) + n - j) * s2;
            double2 q;
            if (VIE) {
                double2 t = cmk(0, 0);
                for (int x = 0; x < S; x++) t = cfma(grow[(long)n * s2 + a * S + x], fr[x * S + b], t);
                q = cfma(cmk(-w, 0.0), t, p.qret[(tri(n) + n - j) * s2 + a * S + b]);
            } else {
                q = a == b ? cneg(cmul(cmk(0.0, poly_diff(k, j, 0) / h), cmk(0.0, -1.0))) : cmk(0, 0);
                q = cadd(q, cmul(cmk(0.0, -w), fr[a * S + b]));
            }
            R[r * S + a] = cconj(q);
        }
    }
    __syncthreads();
    cta_solve(A, R, KS, S, ipiv, status);
    // X_q[a][c] = conj(Y[(q,c), a]) -> G(n, n-q-1)
    for (int e = threadIdx.x; e < k * s2; e += blockDim.x) {
        const int q = e / s2, ac = e % s2, a = ac / S, c = ac % S;
        grow[(long)(n - q - 1) * s2 + ac] = cconj(R[(q * S + c) * S + a]);
    }
    __syncthreads();
}

// les (right solve).  Dyson: unknowns x_j = G^<(j,n), j = 1..k, x_0 = xcol[0] known:
//   sum_m mm(j,m) x_m = gl(j) - (i/h) P(j,0) x_0 + h w(j,0) Sigma^R(j,0) x_0
//   mm(j,m) = (i/h) P(j,m) 1 + delta_jm (mu - H(j)) - h w(j,m) st(j,m)
// VIE2 (vie2_timestep_les, cntr_vie2_impl.hpp:847-990): unknowns j = 0..k:
//   sum_m mm(j,m) x_m = gl(j) + Q^<(j,n),  mm(j,m) = 1 delta_jm + h w(j,m) st(j,m)
// st(j,m) = Sigma^R(j,m) (F^R) for j >= m and -Sigma^R(m,j)^dagger (-Fcc^R) otherwise.
template <int S, bool VIE>
__device__ void les_start_block(const GroupDev &g, const ProbDev &p, int n, const double2 *gl, long ldc, double2 *xcol,
                                double2 *smem) {
    constexpr int j0 = VIE ? 0 : 1;
    const int k = g.k, s2 = S * S, KS = (k + 1 - j0) * S;
    const double h = g.h;
    double2 *A = smem;           // (KS x KS)
    double2 *R = A + KS * KS;    // (KS x S)
    int *ipiv = (int *)(R + KS * S);
    int *status = ipiv + 1;
    if (threadIdx.x == 0) *status = 0;
    for (int e = threadIdx.x; e < KS * (KS + S); e += blockDim.x) {
        const int r = e / (KS + S), c = e % (KS + S), j = r / S + j0, a = r % S;
        if (c < KS) {
            const int m = c / S + j0, b = c % S;
            const double w = h * greg_w(k, j, m);
            const double2 st = j >= m ? g.sret[(tri(j) + m) * s2 + a * S + b]
                                      : cneg(cconj(g.rret[(tri(m) + j) * s2 + b * S + a]));
            double2 v = cscale(st, VIE ? w : -w);
            if (VIE) {
                if (m == j && a == b) v = cadd(v, cmk(1.0, 0.0));
            } else {
                if (a == b) v = cadd(v, cmk(0.0, poly_diff(k, j, m) / h));
                if (m == j) {
                    v = csub(v, p.H[(long)(j + 1) * s2 + a * S + b]);
                    if (a == b) v = cadd(v, cmk(p.mu, 0.0));
                }
            }
            A[r * KS + c] = v;
        } else {
            const int d = c - KS;
            double2 q = gl[((long)j * S + a) * ldc + d];
            if (VIE) {
                q = cadd(q, j <= n ? p.qles[(tri(n) + j) * s2 + a * S + d] : cneg(cconj(p.qles[(tri(j) + n) * s2 + d * S + a])));
            } else {
                const double w = h * greg_w(k, j, 0);
                double2 t = cmk(0, 0);
                for (int b = 0; b < S; b++) t = cfma(g.sret[tri(j) * s2 + a * S + b], xcol[b * S + d], t);
                q = csub(q, cmul(cmk(0.0, poly_diff(k, j, 0) / h), xcol[a * S + d]));
                q = cadd(q, cscale(t, w));
            }
            R[r * S + d] = q;
        }
    }
    __syncthreads();
    cta_solve(A, R, KS, S, ipiv, status);
    for (int e = threadIdx.x; e < KS * S; e += blockDim.x) xcol[j0 * s2 + e] = R[e];
    __syncthreads();
}

// ---------------------------------------------------------------------------------------
// The tv row: G^tv(n, tau) of every problem (dyson_impl :651-741):
//   Q(tau) = sum_{j<n} a_j G^tv(j,tau) + dtau * matsubara_integral_2(Sigma^tv(n,.), G^mat)(tau)
//   G^tv(n,tau) = Minv_les[n] Q(tau)
// The Matsubara integral is linear in G^mat with an operator K_n built from Sigma^tv(n,.)
// alone (k_mat_operator), so for a group sharing Sigma it is one GEMM over all problems
// (Cmat = K_n Gmat_all); these kernels stream the history and add Cmat.  Both work on the device
// layout of G^tv: element planes, (t*s^2 + e)*(ntau+1) + tau, so a warp reading 32 consecutive tau
// of one plane moves 512 contiguous bytes.
// k_tv_ring (FP64 history) and k_tv_mixed (FP32 copy of the history).
// ---------------------------------------------------------------------------------------
// k_tv_ring.  Bound: HBM, the history G^tv(0..n-1) once (size1 >= 6: the FP64 pipe, 8 s flops per
// 16 bytes).  Persistent, one CTA of 16 warps per SM.  A work item is (problem, 32 tau, column d of
// the s x s blocks); warp w takes rows j = w, w + 16, ...  Each warp keeps DEPTH plane rows of 512
// bytes in flight in its own ring in shared memory: a lane copies its 16 bytes with cp.async and
// reads only those, so the ring needs no barrier, and the copies of the next item are issued while
// the current one is still summed.  The coefficients a_j, shared by all items of a group, are
// double-buffered in shared memory and the next chunk waits in registers.  16 x 8 x 512 bytes in
// flight per SM are enough for the full HBM rate; with 64 registers a thread the kernel holds half
// of an SM's registers and a quarter of its shared memory, so that the retarded recursion runs
// beside it (size1 4, 32 problems, n 1200: stream, recursion and les*adv together 3.2 ms, one after
// the other 4.1 ms; size1 1, 1024 problems, n 1000: 2.6 and 2.8 ms); size1 >= 5 takes 128 registers
// and the SM.  Alone: size1 1, 2 6400, 6060 GB/s, size1 4 4280 (register loads, a CTA per 32 tau: 3900),
// size1 8 4010 (1270).  (Loads into registers go through L1 lines, which a shared-memory heavy
// neighbour takes away: 6592 -> 5064 GB/s for size1 1 with the carve-out the recursion needs, and
// without it the two kernels cannot share an SM at all.)
template <int S> struct TvCfg {
    static constexpr int NW = 16, NTH = NW * 32;                       // warps, threads per CTA
    static constexpr int DEPTH = 8;                                    // plane rows in flight per warp
    static constexpr int CHW = S == 1 ? 16 : (S == 2 ? 4 : (S == 3 ? 2 : 1));  // rows per warp and chunk
    static constexpr int CH = CHW * NW, CE = CH * S * S;               // rows, complex of a chunk
    static constexpr int CR = (CE + NTH - 1) / NTH;                    // complex a thread carries to the next
    static constexpr int ring = 0, coef = NW * DEPTH * 32;             // shared memory (complex)
    static constexpr int red = 8 * 32;                                 // partial sums (share the coefficients' place)
    static constexpr int total = coef + (2 * CE > red ? 2 * CE : red);
};
__device__ __forceinline__ void cp16g(double2 *dst, const double2 *src) {  // past L1
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
// Grid (persistent CTAs, groups).  Lanes past ntau copy the previous 32 tau (copies of one address by
// many lanes are slow: size1 1, M 801: 5580 GB/s, so 6400).
template <int S, bool VIE>
__global__ void __launch_bounds__(TvCfg<S>::NTH, S <= 4 ? 2 : 1) k_tv_ring(const GroupDev *__restrict__ gt, GroupSel sel, int n) {
    using C = TvCfg<S>;
    constexpr int s2 = S * S, D = C::DEPTH;
    extern __shared__ double2 rsm_[];
    const GroupDev &g = gt[sel.gid[blockIdx.y]];
    const int M = g.ntau + 1, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tid = threadIdx.x;
    const long rowstride = (long)s2 * M;
    const int ntile = (M + 31) / 32, items = sel.nact[blockIdx.y] * ntile * S;
    if ((int)blockIdx.x >= items) return;
    const int R = n > warp ? (n - warp + C::NW - 1) / C::NW : 0;  // rows of this warp per item
    double2 *ring = rsm_ + C::ring + warp * D * 32 + lane, *cbuf = rsm_ + C::coef;
    const double2 *cf = g.tvcoef;
    // ---- the copy stream of this warp: planes b = 0..S-1 of its rows, item after item
    int lit = R > 0 ? (int)blockIdx.x : items, lrow = 0, lb = 0, lslot = 0;
    const double2 *lptr = nullptr;
    auto open_item = [&]() {
        if (lit >= items) return;
        const int tau = (lit / S) % ntile * 32 + lane;
        lptr = g.probs[lit / (S * ntile)].gtv + (long)warp * rowstride + (long)(lit % S) * M +
               (tau < M ? tau : max(0, tau - 32));
    };
    open_item();
    auto copy_next = [&]() {
        if (lit < items) {
            cp16g(ring + lslot * 32, lptr);
            if (S > 1 && lb < S - 1) {
                lb++;
                lptr += (long)S * M;
            } else {
                lb = 0;
                lptr += C::NW * rowstride - (long)(S - 1) * S * M;
                if (++lrow == R) {
                    lrow = 0;
                    lit += gridDim.x;
                    open_item();
                }
            }
        }
        lslot = lslot + 1 == D ? 0 : lslot + 1;
        cp_commit();  // one group per plane row, empty past the end
    };
#pragma unroll 1
    for (int q = 0; q < D; q++) copy_next();
    int cslot = 0;
    const int nch = (n + C::CH - 1) / C::CH;
    auto coef_at = [&](int ch, int i) {  // complex i of this thread in chunk ch
        const long e = (long)ch * C::CE + tid + (long)i * C::NTH;
        return (tid + i * C::NTH < C::CE && e < (long)n * s2) ? __ldg(cf + e) : cmk(0, 0);
    };
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        double2 acc[S], nx[C::CR];
#pragma unroll
        for (int a = 0; a < S; a++) acc[a] = cmk(0, 0);
#pragma unroll
        for (int i = 0; i < C::CR; i++) nx[i] = coef_at(0, i);
        for (int ch = 0; ch < nch; ch++) {
            double2 *cb = cbuf + (ch & 1) * C::CE;
#pragma unroll
            for (int i = 0; i < C::CR; i++)
                if (tid + i * C::NTH < C::CE) cb[tid + i * C::NTH] = nx[i];
            __syncthreads();  // chunk ch is in place; the other buffer was read before the last barrier
            if (ch + 1 < nch)
#pragma unroll
                for (int i = 0; i < C::CR; i++) nx[i] = coef_at(ch + 1, i);
            const int rows = min(C::CHW, R - ch * C::CHW);
#pragma unroll 1
            for (int r = 0; r < rows; r++) {
                const double2 *cj = cb + (r * C::NW + warp) * s2;
#pragma unroll
                for (int b = 0; b < S; b++) {
                    cp_wait<D - 1>();
                    const double2 x = ring[cslot * 32];
                    cslot = cslot + 1 == D ? 0 : cslot + 1;
#pragma unroll
                    for (int a = 0; a < S; a++) acc[a] = cfma(cj[a * S + b], x, acc[a]);
                    copy_next();
                }
            }
        }
        // sum over the warps, in the place of the coefficients
        __syncthreads();
#pragma unroll
        for (int a = 0; a < S; a++)
#pragma unroll
            for (int half = 8; half > 0; half >>= 1) {
                if (warp >= half && warp < 2 * half) cbuf[(warp - half) * 32 + lane] = acc[a];
                __syncthreads();
                if (warp < half) acc[a] = cadd(acc[a], cbuf[warp * 32 + lane]);
                __syncthreads();
            }
        const int tau = (it / S) % ntile * 32 + lane, d = it % S;
        if (warp == 0 && tau < M) {
            const ProbDev &p = g.probs[it / (S * ntile)];
            // Matsubara part dtau*[c2 + sig c1] from the group GEMM (k_mat_operator)
            const double2 *cm = g.Cmat + (long)tau * S * g.ldc + (long)p.col * S + d;
#pragma unroll
            for (int a = 0; a < S; a++) acc[a] = cadd(acc[a], cm[(long)a * g.ldc]);
            // VIE2 (vie2_timestep_tv, cntr_vie2_impl.hpp:645-725): a_j and Cmat carry the minus sign of
            // the convolution; + Q^tv(n, tau) before the solve with (1 + h w0 F^R(n,n))^-1
            if (VIE) {
                const double2 *qt = p.qtv + (long)n * rowstride + tau;
#pragma unroll
                for (int a = 0; a < S; a++) acc[a] = cadd(acc[a], qt[(long)(a * S + d) * M]);
            }
            const double2 *mi = p.minv_les + (long)n * s2;
#pragma unroll
            for (int a = 0; a < S; a++) {
                double2 x = cmk(0, 0);
#pragma unroll
                for (int b = 0; b < S; b++) x = cfma(mi[a * S + b], acc[b], x);
                p.gtv[(long)n * rowstride + (long)(a * S + d) * M + tau] = x;
            }
        }
    }
    cp_wait<0>();
}

// k_tv_mixed: thread per (tau, column d), a CTA per 32 tau of a problem, 8 warps splitting the rows.
template <int S> struct TvmCfg {
    static constexpr int DCH = S <= 2 ? S : (S <= 4 ? 2 : 1);  // block columns per pass
    static constexpr int NW = 8;                // warps per CTA, splitting the history sum over j
};

// History rows j < n-k-1 are read from the FP32 copy (half the bytes); the k+1 rows
// that carry the backward-difference terms, and all sums, stay in FP64.
// VIE2 (vie2_timestep_tv, cntr_vie2_impl.hpp:645-725): a_j and Cmat carry the minus sign of
// the convolution and Q^tv(n, tau) is added before the solve with (1 + h w0 F^R(n,n))^-1.
template <int S, bool VIE = false>
__global__ void __launch_bounds__(256) k_tv_mixed(const GroupDev *__restrict__ gt, GroupSel sel, int n) {
    constexpr int s2 = S * S, DCH = TvmCfg<S>::DCH, NW = TvmCfg<S>::NW;
    __shared__ double2 red[NW * 32 * S * DCH];
    const GroupDev &g = gt[sel.gid[blockIdx.z]];
    if ((int)blockIdx.y >= sel.nact[blockIdx.z] || (int)blockIdx.x * 32 > g.ntau) return;
    const ProbDev p = g.probs[blockIdx.y];
    const int ntau = g.ntau, M = ntau + 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tau = blockIdx.x * 32 + lane;
    const bool live = tau <= ntau;
    const long rowstride = (long)s2 * M;
    for (int c0 = 0; c0 < S; c0 += DCH) {
        double2 acc[S][DCH];
#pragma unroll
        for (int a = 0; a < S; a++)
#pragma unroll
            for (int c = 0; c < DCH; c++) acc[a][c] = cmk(0, 0);
        if (live) {
            const double2 *gb = p.gtv + tau;
            const double2 *cf = g.tvcoef;
            const int j64 = n - g.k - 1 > 0 ? n - g.k - 1 : 0;  // first FP64 row
            {
                const float2 *gb32 = p.gtv32 + tau;
                // 8-byte loads: twice the rows in flight of the FP64 loop keep as many bytes in flight
#pragma unroll 8
                for (int j = warp; j < j64; j += NW) {
                    const float2 *gj = gb32 + (long)j * rowstride;
                    double2 bv[S][DCH];
#pragma unroll
                    for (int b = 0; b < S; b++)
#pragma unroll
                        for (int c = 0; c < DCH; c++) {
                            float2 f = (c0 + c < S) ? __ldg(gj + (long)(b * S + c0 + c) * M) : make_float2(0.f, 0.f);
                            bv[b][c] = cmk((double)f.x, (double)f.y);
                        }
                    const double2 *cj = cf + (long)j * s2;
#pragma unroll
                    for (int a = 0; a < S; a++)
#pragma unroll
                        for (int b = 0; b < S; b++) {
                            const double2 cab = __ldg(cj + a * S + b);
#pragma unroll
                            for (int c = 0; c < DCH; c++) acc[a][c] = cfma(cab, bv[b][c], acc[a][c]);
                        }
                }
            }
            const int jfirst = j64 + ((warp - j64 % NW) + NW) % NW;  // keep j = warp (mod NW)
#pragma unroll 4
            for (int j = jfirst; j < n; j += NW) {
                const double2 *gj = gb + (long)j * rowstride;
                double2 bv[S][DCH];
#pragma unroll
                for (int b = 0; b < S; b++)
#pragma unroll
                    for (int c = 0; c < DCH; c++)
                        bv[b][c] = (c0 + c < S) ? __ldg(gj + (long)(b * S + c0 + c) * M) : cmk(0, 0);
                const double2 *cj = cf + (long)j * s2;
#pragma unroll
                for (int a = 0; a < S; a++)
#pragma unroll
                    for (int b = 0; b < S; b++) {
                        const double2 cab = __ldg(cj + a * S + b);
#pragma unroll
                        for (int c = 0; c < DCH; c++) acc[a][c] = cfma(cab, bv[b][c], acc[a][c]);
                    }
            }
        }
#pragma unroll
        for (int a = 0; a < S; a++)
#pragma unroll
            for (int c = 0; c < DCH; c++) red[((warp * 32 + lane) * S + a) * DCH + c] = acc[a][c];
        __syncthreads();
        if (warp == 0 && live) {
#pragma unroll
            for (int a = 0; a < S; a++)
#pragma unroll
                for (int c = 0; c < DCH; c++) {
                    double2 v = red[(lane * S + a) * DCH + c];
                    for (int w = 1; w < NW; w++) v = cadd(v, red[((w * 32 + lane) * S + a) * DCH + c]);
                    acc[a][c] = v;
                }
            // Matsubara part dtau*[c2 + sig c1] from the group GEMM (k_mat_operator)
            const double2 *cm = g.Cmat + (long)tau * S * g.ldc + (long)p.col * S + c0;
#pragma unroll
            for (int a = 0; a < S; a++)
#pragma unroll
                for (int c = 0; c < DCH; c++)
                    if (c0 + c < S) acc[a][c] = cadd(acc[a][c], cm[(long)a * g.ldc + c]);
            if (VIE) {
                const double2 *qt = p.qtv + (long)n * rowstride + tau;
#pragma unroll
                for (int a = 0; a < S; a++)
#pragma unroll
                    for (int c = 0; c < DCH; c++)
                        if (c0 + c < S) acc[a][c] = cadd(acc[a][c], qt[(long)(a * S + c0 + c) * M]);
            }
            // solve: G^tv(n,tau)[a][d] = sum_b Minv[a][b] Q[b][d]
            const double2 *mi = p.minv_les + (long)n * s2;
            double2 *out = p.gtv + (long)n * rowstride + tau;
#pragma unroll
            for (int a = 0; a < S; a++)
#pragma unroll
                for (int c = 0; c < DCH; c++) {
                    if (c0 + c >= S) continue;
                    double2 x = cmk(0, 0);
#pragma unroll
                    for (int b = 0; b < S; b++) x = cfma(mi[a * S + b], acc[b][c], x);
                    out[(long)(a * S + c0 + c) * M] = x;
                    p.gtv32[(long)n * rowstride + tau + (long)(a * S + c0 + c) * M] =
                        make_float2((float)x.x, (float)x.y);
                }
        }
        __syncthreads();
    }
}

// k_tv_to32: FP32 copy of G^tv rows [t0, t0+rows) (plane layout, same indexing)
__global__ void k_tv_to32(float2 *__restrict__ dst, const double2 *__restrict__ src, long n) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        dst[i] = make_float2((float)src[i].x, (float)src[i].y);
}

// k_tv_relayout: G^tv between libcntr's layout ((t*M + tau)*s^2 + e) and the element-plane
// layout ((t*s^2 + e)*M + tau) used on the device; rows t = 0..rows-1.
__global__ void k_tv_relayout(double2 *__restrict__ dst, const double2 *__restrict__ src, long rows, int M, int s2,
                              int to_planes) {
    const long total = rows * M * s2;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
        // i indexes the plane layout: t, e, tau
        const long t = i / ((long)s2 * M);
        const int rem = (int)(i % ((long)s2 * M)), e = rem / M, tau = rem % M;
        const long j = (t * M + tau) * s2 + e;  // libcntr index
        if (to_planes) dst[i] = src[j]; else dst[j] = src[i];
    }
}

// ---------------------------------------------------------------------------------------
// One time step t >= 0 between a herm_matrix in device memory and a host slice [ret(t, 0..t) | tv(t, .) |
// les(0..t, t)] in libcntr's layout, one launch: the kernels read / write the host memory themselves
// (pinned, mapped), whole lines at a time.  nrow = (t+1) s^2; planes: tv(t, .) is stored as element
// planes e (ntau+1) + tau (a tile of 32 tau goes through shared memory), else in libcntr's layout; tv32:
// FP32 copy of the tv row, or null.  Grid: 2 ceil(nrow / 1024) + slice_tv_blocks, 256 threads.
// ---------------------------------------------------------------------------------------
__host__ __device__ inline int slice_row_blocks(long nrow) { return (int)((nrow + 1023) / 1024); }
__host__ __device__ inline int slice_tv_blocks(int M, int s2, int planes) {
    return planes && s2 > 1 ? (M + 31) / 32 : (int)(((long)M * s2 + 1023) / 1024);
}
template <bool PACK>
__global__ void __launch_bounds__(256) k_slice(double2 *host, double2 *ret, double2 *tv, double2 *les, float2 *tv32,
                                               long nrow, int M, int s2, int planes) {
    __shared__ double2 sm[32 * NESSI_MAXS * NESSI_MAXS];
    const int nb = slice_row_blocks(nrow), blk = blockIdx.x, tid = threadIdx.x;
    auto move = [&](double2 *dev, double2 *h, long n, long c0) {
        double2 v[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const long x = c0 + tid + 256 * i;
            if (x < n) v[i] = PACK ? dev[x] : h[x];
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const long x = c0 + tid + 256 * i;
            if (x < n) (PACK ? h : dev)[x] = v[i];
        }
    };
    auto to32 = [](double2 v) { return make_float2((float)v.x, (float)v.y); };
    if (blk < nb) {
        move(ret, host, nrow, blk * 1024L);
    } else if (blk < 2 * nb) {
        move(les, host + nrow + (long)M * s2, nrow, (blk - nb) * 1024L);
    } else if (!planes || s2 == 1) {
        const long c0 = (blk - 2 * nb) * 1024L, n = (long)M * s2;
        move(tv, host + nrow, n, c0);
        if (!PACK && tv32)
            for (long x = c0 + tid; x < n && x < c0 + 1024; x += 256) tv32[x] = to32(tv[x]);
    } else {
        const int tau0 = (blk - 2 * nb) * 32, cnt = min(32, M - tau0);
        double2 *h = host + nrow + (long)tau0 * s2;
        if (!PACK) {
            for (int x = tid; x < cnt * s2; x += 256) sm[x] = h[x];
            __syncthreads();
        }
        for (int x = tid; x < 32 * s2; x += 256) {
            const int e = x / 32, l = x % 32;
            if (l >= cnt) continue;
            const long i = (long)e * M + tau0 + l;
            if (PACK) {
                sm[l * s2 + e] = tv[i];
            } else {
                tv[i] = sm[l * s2 + e];
                if (tv32) tv32[i] = to32(sm[l * s2 + e]);
            }
        }
        if (PACK) {
            __syncthreads();
            for (int x = tid; x < cnt * s2; x += 256) h[x] = sm[x];
        }
    }
}

// ---------------------------------------------------------------------------------------
// k_mat_operator: K_n[(m,a),(x,c)] such that dtau * matsubara_integral_2(Sigma^tv(n,.), B)(m)
// = sum_x K_n[m,x] B(x) for every B (conv_impl :410-540 read as a linear map of B):
//   c2 = sum_{l=0}^{r} w(r,l) A(m+l) B(l)           (r = ntau-m >= k; rcorr for 0<r<k)
//   c1 = sum_{l=0}^{m} w(m,l) A(m-l) B(ntau-l)      (m >= k; rcorr for 0<m<k),  C = c2 + sig c1
// ---------------------------------------------------------------------------------------
// (conv_sign = -1 for VIE2, whose Matsubara convolution enters the right-hand side with a minus sign.)
template <int S>
__global__ void k_mat_operator(const GroupDev *__restrict__ gt, GroupSel sel, int n) {
    pdl_entry();
    const GroupDev &g = gt[sel.gid[blockIdx.y]];
    const int k = g.k, s2 = S * S, ntau = g.ntau, M = ntau + 1;
    const long KS = (long)M * S;
    const double2 *A = g.stv + (long)n * M * s2;
    const double dtau = g.beta / ntau, sg = (double)g.sig;
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < (long)M * M * s2; e += (long)gridDim.x * blockDim.x) {
        const int m = (int)(e / ((long)M * s2));
        const int rem = (int)(e % ((long)M * s2));
        const int x = rem / s2, ac = rem % s2, a = ac / S, c = ac % S;
        const int r = ntau - m;
        double2 v = cmk(0, 0);
        if (r >= k) {
            if (x <= r) v = cfma(cmk(greg_w(k, r, x), 0), A[(long)(m + x) * s2 + ac], v);
        } else if (r > 0 && x <= k) {
            for (int l = 0; l <= k; l++) v = cfma(cmk(rcorr_w(k, r, l, x), 0), A[(long)(ntau - l) * s2 + ac], v);
        }
        const int l = ntau - x;
        if (m >= k) {
            if (l >= 0 && l <= m) v = cfma(cmk(sg * greg_w(k, m, l), 0), A[(long)(m - l) * s2 + ac], v);
        } else if (m > 0 && l >= 0 && l <= k) {
            for (int jj = 0; jj <= k; jj++) v = cfma(cmk(sg * rcorr_w(k, m, l, jj), 0), A[(long)jj * s2 + ac], v);
        }
        g.Kmat[((long)m * S + a) * KS + (long)x * S + c] = cscale(v, dtau * g.conv_sign);
    }
}

// k_gmat_stack: Gmat_all[(x,c)][(col,d)] = G^mat_col(x)[c][d]
template <int S>
__global__ void k_gmat_stack(GroupDev g, const ProbDev *__restrict__ probs) {
    const ProbDev p = probs[blockIdx.y];
    const int s2 = S * S, M = g.ntau + 1;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < M * s2; e += gridDim.x * blockDim.x) {
        const int x = e / s2, cd = e % s2, c = cd / S, d = cd % S;
        g.Gmat_all[((long)x * S + c) * g.ldc + (long)p.col * S + d] = p.gmat[e];
    }
}

// ---------------------------------------------------------------------------------------
// k_les_operands_t: right-hand operand of the Sigma-shared product tv*vt (conv_impl :1075-1242)
//   btv [(m,c)][(col,d)] = w(ntau,m) (-i dtau)(-sig) G^tv(n,ntau-m)^dagger[c][d]
// (badv[(m,c)][(col,d)] = h w(n,m) G^R(n,m)^dagger[c][d] comes from the retarded recursion).  btv is
// row-major with the problems side by side in a row, so one problem's column is a strided write; a
// CTA takes a tile of LOT problems x LOR time indices, reads each problem's contiguous slice into
// shared memory and writes whole row segments (coalesced).
// ---------------------------------------------------------------------------------------
#define LOT 32
template <int S> struct LoCfg {
    static constexpr int LOR = S == 1 ? 32 : (S == 2 ? 16 : (S <= 4 ? 4 : 1));  // time indices per tile
};

template <int S>
__global__ void __launch_bounds__(256) k_les_operands_t(const GroupDev *__restrict__ gt, GroupSel sel, int n) {
    constexpr int s2 = S * S, LOR = LoCfg<S>::LOR;
    pdl_entry();
    const GroupDev &g = gt[sel.gid[blockIdx.z]];
    const ProbDev *probs = g.probs;
    const int nact = sel.nact[blockIdx.z];
    if ((int)blockIdx.y * LOT >= nact || (int)blockIdx.x * LOR > g.ntau) return;
    __shared__ double2 buf[LOT * LOR * s2 + LOT];
    __shared__ const double2 *src[LOT];
    __shared__ int colid[LOT];
    const int k = g.k, ntau = g.ntau, M = ntau + 1;
    const double dtau = g.beta / ntau;
    const long ldc = g.ldc;
    const int q0 = blockIdx.y * LOT, nq = min(LOT, nact - q0);
    const int m0 = blockIdx.x * LOR, nm = min(LOR, M - m0);
    if (threadIdx.x < LOT) {
        const int q = threadIdx.x;
        src[q] = q < nq ? probs[q0 + q].gtv + (long)n * s2 * M : nullptr;
        colid[q] = q < nq ? probs[q0 + q].col : 0;
    }
    __syncthreads();
    // gather: buf[(q*LOR + mm)*s2 + e] = G^tv element e of problem q at tau index ntau - (m0+mm)
    for (int i = threadIdx.x; i < nq * nm * s2; i += blockDim.x) {
        const int q = i / (nm * s2), rem = i % (nm * s2), e = rem / nm, mm = rem % nm;
        buf[(q * LOR + mm) * s2 + e] = src[q][(long)e * M + (ntau - (m0 + mm))];  // tv planes
    }
    __syncthreads();
    // scatter: row (m, c), columns (col, d) of this tile
    for (int i = threadIdx.x; i < nm * S * nq * S; i += blockDim.x) {
        const int r = i / (nq * S), cc = i % (nq * S), mm = r / S, c = r % S, q = cc / S, d = cc % S;
        const int m = m0 + mm;
        const double2 v = cconj(buf[(q * LOR + mm) * s2 + d * S + c]);
        g.btv[((long)m * S + c) * ldc + (long)colid[q] * S + d] =
            cmul(cmk(0.0, dtau * (double)g.sig * greg_w(k, ntau, m)), v);
    }
}

// ---------------------------------------------------------------------------------------
// The three Sigma-shared products of a step, one launch for all selected groups (grid z):
//   PROD_MAT     Cmat = K_n Gmat_all                        (Matsubara part of the tv row)
//   PROD_LESADV  gles = +- Sigma^<_dense badv               (les*adv)
//   PROD_TVVT    gles += +- Sigma^tv btv                    (tv*vt)
// ---------------------------------------------------------------------------------------
enum { PROD_MAT, PROD_LESADV, PROD_TVVT };
struct ProdDims {
    int M, N, K;
};
template <int OP>
__host__ __device__ inline ProdDims prod_dims(int s, int ntau, int n, int nact) {
    const int MS = (ntau + 1) * s, nn = (n + 1) * s;
    return ProdDims{OP == PROD_MAT ? MS : nn, nact * s, OP == PROD_LESADV ? nn : MS};
}
template <int OP>
__host__ __device__ inline ProdDims prod_operands(const GroupDev &g, int n, int nact, LdRowK &la, LdRowN &lb, StRow &st) {
    const ProdDims d = prod_dims<OP>(g.s, g.ntau, n, nact);
    const long ldL = (long)(g.ntmax + 1) * g.s, MS = (long)(g.ntau + 1) * g.s;
    if (OP == PROD_MAT) {
        la = LdRowK{g.Kmat, MS, d.M, d.K};
        lb = LdRowN{g.Gmat_all, g.ldc, d.K, d.N};
        st = StRow{g.Cmat, g.ldc, d.M, d.N, 1.0, 0};
    } else if (OP == PROD_LESADV) {
        la = LdRowK{g.Ldense, ldL, d.M, d.K};
        lb = LdRowN{g.badv, g.ldc, d.K, d.N};
        st = StRow{g.gles, g.ldc, d.M, d.N, g.conv_sign, 0};
    } else {
        la = LdRowK{g.s == 1 ? g.stv : g.Tdense, MS, d.M, d.K};
        lb = LdRowN{g.btv, g.ldc, d.K, d.N};
        st = StRow{g.gles, g.ldc, d.M, d.N, g.conv_sign, 1};
    }
    return d;
}
template <int OP>
__global__ void __launch_bounds__(128, 4) k_zgemm(const GroupDev *__restrict__ gt, GroupSel sel, int n) {
    extern __shared__ double2 zsm[];
    LdRowK la;
    LdRowN lb;
    StRow st;
    pdl_entry();
    const ProdDims d = prod_operands<OP>(gt[sel.gid[blockIdx.z]], n, sel.nact[blockIdx.z], la, lb, st);
    if ((int)blockIdx.y * 32 >= d.M || (int)blockIdx.x * 32 >= d.N) return;
    zgemm_pipe<32, 32>(la, lb, st, blockIdx.y * 32, blockIdx.x * 32, d.K, zsm);
}
template <int OP>
__global__ void __launch_bounds__(256, 2) k_zgemm_split(const GroupDev *__restrict__ gt, GroupSel sel, int n) {
    __shared__ double2 red[8 * 32 * 8];
    LdRowK la;
    LdRowN lb;
    StRow st;
    pdl_entry();
    const ProdDims d = prod_operands<OP>(gt[sel.gid[blockIdx.z]], n, sel.nact[blockIdx.z], la, lb, st);
    if ((int)blockIdx.y * 32 >= d.M || (int)blockIdx.x * 8 >= d.N) return;
    zgemm_split(la, lb, st, blockIdx.y * 32, blockIdx.x * 8, d.K, red);
}
// one group: the operands in the kernel's parameters (2002 x 512 x 2002 521 us, through the table 542)
__global__ void __launch_bounds__(256, 2) k_zgemm_split1(LdRowK la, LdRowN lb, StRow st, int K) {
    __shared__ double2 red[8 * 32 * 8];
    pdl_entry();
    zgemm_split(la, lb, st, blockIdx.y * 32, blockIdx.x * 8, K, red);
}
