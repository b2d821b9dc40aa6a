/*
 * Cholesky of a 128 x 128 block held in shared memory by one CTA, with the
 * inverses of its diagonal blocks, log-det and the forward solve of a
 * right-hand side; used by the sub-block POTRF kernel and the tile DAG kernel.
 */
#ifndef EXAGEOSTAT_B200_POTRF128_CUH
#define EXAGEOSTAT_B200_POTRF128_CUH

#include "xg_common.cuh"

#define XG_SUB 128
#define XG_P_NB 16             /* panel width inside the sub-block */
#define XG_P_LDS (XG_SUB + 4) /* DMMA operand reads: g * 2 * 132 = 8 g (mod 32 banks), conflict-free */
#define XG_P_LDW (XG_P_NB + 4)
#define XG_P_WSZ (XG_P_NB * XG_P_LDW)
#define XG_POTRF_SUB_THREADS 256
/* doubles of shared memory of xg_potrf128: [128][132] block, [8][16][20] inverses, [2][16][20] scratch, [128] rhs */
#define XG_P_DOUBLES (XG_SUB * XG_P_LDS + (XG_SUB / XG_P_NB + 2) * XG_P_WSZ + XG_SUB)

/* 1 / sqrt(d): the hardware's approximation y (rsqrt.approx.ftz.f64, measured
 * within 2^-20) and one step of Householder's third-order iteration,
 * y (1 + e / 2 + 3 e^2 / 8) with e = 1 - d y^2, whose own error is 5/16 e^3 <
 * 2^-58; measured within 1.25 x 2^-53 relative of 1 / sqrt(d).  Shorter than
 * rsqrt() and without its branch, so a caller's independent work schedules
 * around it.  For normal d (xg_p_in_range). */
__device__ __forceinline__ double xg_rsqrt_fast(double d)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = fma(-d * y, y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}
/* 2^-967 <= d < 2^967, from the high word: one integer comparison that also
 * refuses zero, negative numbers, infinities and NaN */
__device__ __forceinline__ bool xg_p_in_range(double d)
{
    return (unsigned)__double2hiint(d) - 0x03800000u < 0x78E00000u;
}

/* Cholesky of a 16 x 16 block by one warp, with its inverse: lane r < 16 holds
 * row r of the block, lane 16 + r row r of the identity (W holds it on entry).
 * The right-looking column operations that turn the block into L turn the
 * identity rows into L^-T in the same instructions.  The pivots never leave
 * the lanes: with alpha = a(j+1, j+1) and beta = a(j+1, j) broadcast while the
 * reciprocal root of d_j is under way, every lane forms d_{j+1} = alpha -
 * L(j+1, j)^2 itself, so the chain per column is the reciprocal root, a
 * product and an FMA.  The column just scaled reaches the other lanes through
 * shared memory (two doubles a load of 9 cycles; a double costs two shuffles
 * of 4).  Nothing is selected or tested inside the loop (that alone cost 1500
 * of 3500 cycles): entries above the diagonal come out meaningless, and the
 * pivots are examined after it.
 * S (leading dimension XG_P_LDS) receives L (rows' entries right of the
 * diagonal undefined), W L^-T; buf: 64 doubles, 16-byte aligned.  FAST returns
 * -1, with nothing written to S and W, when a pivot is not a positive number
 * of ordinary size; the other form returns the first column (1-based) whose
 * pivot is not positive, or 0, in every lane. */
template <bool FAST>
__device__ __forceinline__ int xg_chol16_pass(double *S, double *W, double *buf, int lane)
{
    const int r = lane & 15;
    const bool ident = lane >= 16;
    double *row = ident ? W + r * XG_P_LDW : S + r * XG_P_LDS;
    double2 *piv = reinterpret_cast<double2 *>(buf + 2 * XG_P_NB); /* [16] (d_j, 1 / sqrt(d_j)) */
    double a[XG_P_NB];
#pragma unroll
    for (int c = 0; c < XG_P_NB; c += 2) {
        const double2 v = *reinterpret_cast<const double2 *>(row + c);
        a[c] = v.x;
        a[c + 1] = v.y;
    }
    int fail = 0;
    double d = __shfl_sync(0xffffffffu, a[0], 0);
#pragma unroll
    for (int j = 0; j < XG_P_NB; ++j) {
        double alpha = 0.0, beta = 0.0;
        if (j + 1 < XG_P_NB) {
            beta = __shfl_sync(0xffffffffu, a[j], j + 1);
            alpha = __shfl_sync(0xffffffffu, a[j + 1], j + 1);
        }
        if (!FAST) {
            const bool bad = !(d > 0.0);
            fail = bad && !fail ? j + 1 : fail;
            d = bad ? 1.0 : d;
        }
        const double ri = FAST ? xg_rsqrt_fast(d) : rsqrt(d);
        piv[j] = make_double2(d, ri);
        a[j] *= ri;
        if (j + 1 < XG_P_NB) {
            const double lb = beta * ri; /* L(j+1, j), as lane j + 1 forms it */
            d = fma(-lb, lb, alpha);
            a[j + 1] = fma(-a[j], lb, a[j + 1]);
        }
        if (j + 2 < XG_P_NB) {
            /* entries j + 2 .. 15 of the column; two buffers, so a column's
             * stores never meet the loads of the one before */
            double *col = buf + (j & 1) * XG_P_NB;
            if (!ident) col[r] = a[j];
            __syncwarp();
#pragma unroll
            for (int c = (j + 2) & ~1; c < XG_P_NB; c += 2) {
                const double2 v = *reinterpret_cast<const double2 *>(col + c);
                if (c >= j + 2) a[c] = fma(-a[j], v.x, a[c]);
                a[c + 1] = fma(-a[j], v.y, a[c + 1]);
            }
        }
    }
    __syncwarp();
    const double2 pr = piv[r];
    if (FAST && !__all_sync(0xffffffffu, xg_p_in_range(pr.x))) return -1;
#pragma unroll
    for (int c = 0; c < XG_P_NB; c += 2) *reinterpret_cast<double2 *>(row + c) = make_double2(a[c], a[c + 1]);
    /* L_rr = d ri with one Newton correction of the square root */
    const double l0 = pr.x * pr.y;
    if (!ident) row[r] = fma(fma(-l0, l0, pr.x), 0.5 * pr.y, l0);
    return fail;
}

/* the general form: kept out of line, it runs only for the odd block whose
 * pivots are out of range or not positive */
static __device__ __noinline__ int xg_chol16_general(double *S, double *W, double *buf, int lane)
{
    return xg_chol16_pass<false>(S, W, buf, lane);
}

__device__ __forceinline__ int xg_chol16_warp(double *S, double *W, double *buf, int lane)
{
    const int f = xg_chol16_pass<true>(S, W, buf, lane);
    return f >= 0 ? f : xg_chol16_general(S, W, buf, lane);
}

/* The panel products run as m16n8k4 DMMAs whose eight columns n stand for the
 * block's columns pi(n) = 0, 6, 1, 7, 2, 4, 3, 5: a lane's two results are
 * then columns tq and 4 + (tq + 2) % 4, and with row strides of 4 (mod 16)
 * doubles the operand reads (rows g or pi(g), columns tq) and the 8-byte
 * result accesses all touch 32 distinct banks per half warp. */
__device__ __forceinline__ int xg_p_perm(int g) { return g & 1 ? 4 + (((g >> 1) + 2) & 3) : g >> 1; }
__device__ __forceinline__ int xg_p_col(int e, int tq) { return e ? 4 + ((tq + 2) & 3) : tq; }

/* acc (16 x 16: two 16 x 8 DMMA tiles) += A B over K = 16 for one warp, A(r, k)
 * = a[r lda + k]; B(k, n) = b[k ldb + n] (BT false) or b[n ldb + k] (BT true),
 * all in shared memory. */
template <bool BT>
__device__ __forceinline__ void xg_mma16(double (&acc)[2][4], const double *a, int lda, const double *b, int ldb,
                                         int g, int tq)
{
    const int pg = xg_p_perm(g);
    double av[4][2], bv[4][2];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        av[k][0] = a[g * lda + 4 * k + tq];
        av[k][1] = a[(g + 8) * lda + 4 * k + tq];
#pragma unroll
        for (int n = 0; n < 2; ++n)
            bv[k][n] = BT ? b[(n * 8 + pg) * ldb + 4 * k + tq] : b[(4 * k + tq) * ldb + n * 8 + pg];
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int n = 0; n < 2; ++n)
            xg_dmma_16x8x4(acc[n][0], acc[n][1], acc[n][2], acc[n][3], av[k][0], av[k][1], bv[k][n]);
}

/* NH 16 x 8 halves (columns 8 n0 ..) of block row i, one warp: column q = p + 1
 * by panel p, column q + 1 by the panels 0 .. p,
 *   S_iq -= X_ip X_qp^T,   S_i,q+1 -= sum_{k <= p} X_ik X_{q+1,k}^T,
 * in one call, so that the chains of dependent DMMAs overlap and panel p's
 * rows of X are read once. */
template <int NH>
__device__ __forceinline__ void xg_potrf_update(double *S, int i, int p, int n0, int g, int tq)
{
    const int q = p + 1, pg = xg_p_perm(g);
    double *c0 = S + (i * XG_P_NB + g) * XG_P_LDS + q * XG_P_NB + n0 * 8;
    const double *a = S + (i * XG_P_NB + g) * XG_P_LDS + tq;
    const double *b = S + (q * XG_P_NB + n0 * 8 + pg) * XG_P_LDS + tq;
    double cq[NH][4], cn[NH][4]; /* start at -S, stored negated */
#pragma unroll
    for (int n = 0; n < NH; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const double *c = c0 + 8 * (e >> 1) * XG_P_LDS + n * 8 + xg_p_col(e & 1, tq);
            cq[n][e] = -c[0];
            cn[n][e] = -c[XG_P_NB];
        }
    for (int k = p; k >= 0; --k) {
        double a0[4], a1[4], bn[NH][4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            a0[s] = a[k * XG_P_NB + 4 * s];
            a1[s] = a[8 * XG_P_LDS + k * XG_P_NB + 4 * s];
#pragma unroll
            for (int n = 0; n < NH; ++n) bn[n][s] = b[(XG_P_NB + 8 * n) * XG_P_LDS + k * XG_P_NB + 4 * s];
        }
        if (k == p) {
            double bq[NH][4];
#pragma unroll
            for (int s = 0; s < 4; ++s)
#pragma unroll
                for (int n = 0; n < NH; ++n) bq[n][s] = b[8 * n * XG_P_LDS + k * XG_P_NB + 4 * s];
#pragma unroll
            for (int s = 0; s < 4; ++s)
#pragma unroll
                for (int n = 0; n < NH; ++n) {
                    xg_dmma_16x8x4(cq[n][0], cq[n][1], cq[n][2], cq[n][3], a0[s], a1[s], bq[n][s]);
                    xg_dmma_16x8x4(cn[n][0], cn[n][1], cn[n][2], cn[n][3], a0[s], a1[s], bn[n][s]);
                }
        } else {
#pragma unroll
            for (int s = 0; s < 4; ++s)
#pragma unroll
                for (int n = 0; n < NH; ++n)
                    xg_dmma_16x8x4(cn[n][0], cn[n][1], cn[n][2], cn[n][3], a0[s], a1[s], bn[n][s]);
        }
    }
#pragma unroll
    for (int n = 0; n < NH; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            double *c = c0 + 8 * (e >> 1) * XG_P_LDS + n * 8 + xg_p_col(e & 1, tq);
            c[0] = -cq[n][e];
            c[XG_P_NB] = -cn[n][e];
        }
}

/* Block row p + 1 of panel p and the next diagonal block, by one warp: X = B W
 * to S, then the caller's signal, then S_{p+1,p+1} -= X X^T.  The second
 * product takes both operands from the first one's accumulators: with the K
 * index running over the columns in the order the lanes hold them, the
 * fragment of X as A is that of X^T as B. */
template <typename Signal>
__device__ __forceinline__ void xg_potrf_next_diag(double *S, const double *W, int p, int g, int tq, Signal signal)
{
    double *B = S + (p + 1) * XG_P_NB * XG_P_LDS + p * XG_P_NB;
    double2 *C = reinterpret_cast<double2 *>(S + ((p + 1) * XG_P_NB + g) * XG_P_LDS + (p + 1) * XG_P_NB + 2 * tq);
    double c[2][4]; /* columns 2 tq, 2 tq + 1 of either half, negated */
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const double2 v = C[h * 4 * XG_P_LDS + n * 4];
            c[n][2 * h] = -v.x;
            c[n][2 * h + 1] = -v.y;
        }
    double x[2][4] = {{0.0, 0.0, 0.0, 0.0}, {0.0, 0.0, 0.0, 0.0}};
    xg_mma16<false>(x, B, XG_P_LDS, W, XG_P_LDW, g, tq);
    __syncwarp();
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) B[(g + 8 * (e >> 1)) * XG_P_LDS + n * 8 + xg_p_col(e & 1, tq)] = x[n][e];
    signal();
#pragma unroll
    for (int k = 0; k < 4; ++k) { /* columns xg_p_col(k & 1) of half k / 2 */
        const double x0 = x[k >> 1][k & 1], x1 = x[k >> 1][2 + (k & 1)];
        xg_dmma_16x8x4(c[0][0], c[0][1], c[0][2], c[0][3], x0, x1, x0);
        xg_dmma_16x8x4(c[1][0], c[1][1], c[1][2], c[1][3], x0, x1, x1);
    }
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) C[h * 4 * XG_P_LDS + n * 4] = make_double2(-c[n][2 * h], -c[n][2 * h + 1]);
    __syncwarp();
}

/* out (16 x 16, leading dimension ldo) = s A B, K = 16 (one warp) */
template <bool BT>
__device__ __forceinline__ void xg_potrf_product16(double *out, int ldo, double s, const double *a, int lda,
                                                   const double *b, int ldb, int g, int tq)
{
    double acc[2][4] = {{0.0, 0.0, 0.0, 0.0}, {0.0, 0.0, 0.0, 0.0}};
    xg_mma16<BT>(acc, a, lda, b, ldb, g, tq);
    __syncwarp();
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) out[(g + 8 * (e >> 1)) * ldo + n * 8 + xg_p_col(e & 1, tq)] = s * acc[n][e];
}

/* The inverse of the 32 x 32 diagonal block b of L from those of its 16 x 16
 * ones (one warp; scratch T: [2][16][20]): [[D11, 0], [-D22 L21 D11, D22]],
 * D = W^T, to D[i * 32 + c]. */
__device__ __forceinline__ void xg_potrf_inverse32(const double *S, const double *W, double *T, int b, double *D,
                                                   int lane)
{
    const int g = lane >> 2, tq = lane & 3;
    const double *W1 = W + 2 * b * XG_P_WSZ, *W2 = W1 + XG_P_WSZ;
    double *T2 = T + XG_P_WSZ;
    /* L21 D11: B(k, n) = D11(k, n) = W1(n, k); D22 = W2^T beside it */
    xg_potrf_product16<true>(T, XG_P_LDW, 1.0, S + (32 * b + 16) * XG_P_LDS + 32 * b, XG_P_LDS, W1, XG_P_LDW, g, tq);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        const int idx = u * 32 + lane, i = idx >> 4, c = idx & 15;
        const double d2 = W2[c * XG_P_LDW + i];
        T2[i * XG_P_LDW + c] = d2;
        D[i * 32 + c] = W1[c * XG_P_LDW + i];
        D[i * 32 + 16 + c] = 0.0;
        D[(16 + i) * 32 + 16 + c] = d2;
    }
    __syncwarp();
    xg_potrf_product16<false>(D + 16 * 32, 32, -1.0, T2, XG_P_LDW, T, XG_P_LDW, g, tq);
    __syncwarp();
}

/* Cholesky of the 128 x 128 block in S by one CTA of 256 threads, in eight
 * 16-wide panels: per panel warp 0 factors the diagonal block and inverts it
 * (xg_chol16_warp); each block row below is multiplied by the inverse on DMMA
 * (one warp each); warp 0 goes on with the next diagonal block -- its last
 * update needs only the block row warp 0 itself solved -- and factors it.
 * Meanwhile six warps finish the next block column (the update by the panel
 * just solved) and bring the one after it up to date (all earlier panels):
 * left-looking, so every stage has 12 to 16 products and none is longer than
 * the factorisation it hides behind (right-looking, the first two had 27 and
 * 20, and the chain waited for them).  The serial chain is 8 x (16 pivots +
 * two 16 x 16 products).  Warp 4, which shares warp 0's scheduler, takes what
 * is light on the FP64 pipe: the forward solve of the right-hand side vs
 * (rhs) and the finished block column to the global tile Lg (leading
 * dimension ldl, zeros above the diagonal); warp 7 forms the inverted 32 x 32
 * diagonal blocks (dinv), warp 5 the logarithms.
 * W keeps the inverses L_pp^-T; sums[0] = sum log L_ii, sums[1] = |vs|^2
 * after the solve (shared memory).  Returns the first failing column
 * (1-based) or 0 to every thread; L, vs, W and sums are complete and visible
 * to all then.
 *
 * A latency chain of 128 pivots on one SM bounds it. */
__device__ __forceinline__ int xg_potrf128(double *S, double *W, double *T, double *vs, int rhs, double *Lg, int ldl,
                                           double *dinv, double *sums)
{
    /* warp 0 runs ahead into panel p + 1 while the others may still be about to
     * read panel p's word: two words in turn, so that a word is written again
     * only behind the barrier of the panel between */
    __shared__ int s_fail[2];
    __shared__ __align__(16) double s_buf[4 * XG_P_NB];
    constexpr int NP = XG_SUB / XG_P_NB;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, tq = lane & 3;
    if (tid < 2) s_fail[tid] = 0;
    for (int idx = tid; idx < NP * XG_P_NB * XG_P_NB; idx += XG_POTRF_SUB_THREADS) {
        const int r = (idx >> 4) & 15, c = idx & 15;
        W[(idx >> 8) * XG_P_WSZ + r * XG_P_LDW + c] = r == c ? 1.0 : 0.0;
    }
    double mine = 0.0; /* warp 4: |vs|^2, warp 5: log-det, by lane */
    __syncthreads();
#pragma unroll 1
    for (int p = 0; p < NP; ++p) {
        const int c0 = p * XG_P_NB;
        const double *Wp = W + p * XG_P_WSZ;
        if (warp == 0) {
            const int f = xg_chol16_warp(S + c0 * XG_P_LDS + c0, W + p * XG_P_WSZ, s_buf, lane);
            if (f && lane == 0) s_fail[p & 1] = c0 + f;
        }
        __syncthreads();
        const int failed = s_fail[p & 1];
        if (failed) return failed;
        if (warp == 0) {
            if (p + 1 < NP)
                xg_potrf_next_diag(S, Wp, p, g, tq, [] {
                    __threadfence_block();
                    asm volatile("bar.arrive 1, 256;" ::: "memory"); /* block row p + 1 is solved */
                });
        } else if (warp == 4) {
            if (rhs) { /* w = L_pp^-1 vs_p: (vs_p^T W)_c, lane c */
                double w = 0.0;
                if (lane < XG_P_NB)
#pragma unroll
                    for (int r = 0; r < XG_P_NB; ++r) w = fma(vs[c0 + r], Wp[r * XG_P_LDW + lane], w);
                __syncwarp();
                if (lane < XG_P_NB) vs[c0 + lane] = w;
                mine = fma(w, w, mine);
            }
            if (p + 1 < NP) asm volatile("bar.sync 1, 256;" ::: "memory");
            if (rhs) {
                __syncwarp();
                double w[XG_P_NB];
#pragma unroll
                for (int c = 0; c < XG_P_NB; ++c) w[c] = vs[c0 + c];
                for (int r = c0 + XG_P_NB + lane; r < XG_SUB; r += 32) {
                    double t = vs[r];
#pragma unroll
                    for (int c = 0; c < XG_P_NB; c += 2) {
                        const double2 x = *reinterpret_cast<const double2 *>(S + r * XG_P_LDS + c0 + c);
                        t = fma(-x.x, w[c], t);
                        t = fma(-x.y, w[c + 1], t);
                    }
                    vs[r] = t;
                }
            }
            const int c = c0 + 2 * (lane & 7);
#pragma unroll 4
            for (int r = lane >> 3; r < XG_SUB; r += 4) {
                double2 x = *reinterpret_cast<const double2 *>(S + r * XG_P_LDS + c);
                if (c > r) x.x = 0.0;
                if (c + 1 > r) x.y = 0.0;
                *reinterpret_cast<double2 *>(Lg + (long long)r * ldl + c) = x;
            }
        } else {
            const int w6 = warp < 4 ? warp - 1 : warp - 2;
            if (p + 1 < NP) {
                const int i0 = p + 2 + w6;
                if (i0 < NP) {
                    double *B = S + i0 * XG_P_NB * XG_P_LDS + c0;
                    xg_potrf_product16<false>(B, XG_P_LDS, 1.0, B, XG_P_LDS, Wp, XG_P_LDW, g, tq);
                }
                asm volatile("bar.sync 1, 256;" ::: "memory");
                /* block rows i > q = p + 1, a warp each; of three rows or fewer, half a row each */
                const int rows = NP - 2 - p;
                if (rows > 3) {
                    if (w6 < rows) xg_potrf_update<2>(S, p + 2 + w6, p, 0, g, tq);
                } else if (w6 < 2 * rows) {
                    xg_potrf_update<1>(S, p + 2 + (w6 >> 1), p, w6 & 1, g, tq);
                }
            }
            if (dinv && warp == 7 && (p & 1)) xg_potrf_inverse32(S, W, T, p >> 1, dinv + (p >> 1) * 32 * 32, lane);
            if (warp == 5 && lane < XG_P_NB) mine += log(S[(c0 + lane) * (XG_P_LDS + 1)]);
        }
    }
    if (warp == 4 || warp == 5) {
        double t = lane < XG_P_NB ? mine : 0.0;
        for (int off = 8; off > 0; off >>= 1) t += __shfl_xor_sync(0xffffffffu, t, off);
        if (lane == 0) sums[warp == 4] = t;
    }
    __syncthreads();
    return 0;
}

#endif
