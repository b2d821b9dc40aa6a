/*
 * Assessment of a fitted model, on sm_100a: the Fisher information matrix and
 * the MLOE / MMOM criteria.
 *
 * Fisher (EXAGEOSTAT_Fisher_Tile, exageostat_exact/src/compute/MLE_dexact.c:1777-1934):
 *   F_jk = 1/2 tr(Sigma^-1 dSigma_j Sigma^-1 dSigma_k), then F^-1.
 *   The reference forms Sigma^-1 dSigma_j by two N x N triangular solves per
 *   (j, k) pair and multiplies the pairs (30 N^3 flops for three parameters).
 *   Here tr(Sigma^-1 D_j Sigma^-1 D_k) = <W_j, W_k> with the symmetric
 *   W_j = L^-1 D_j L^-T: Y_j = D_j L^-T are the rows Y_j L^T = D_j (N^3 flops),
 *   and the lower half of W_j the rows W_j L^T = Y_j^T (N^3 / 3), all j in one
 *   dataflow launch each (rows_dag.cu), then one pass over the W_j
 *   (xg_fisher_trace_kernel).  dSigma_sigma^2 = (Sigma - tau^2 I) / sigma^2
 *   gives W = (I - tau^2 M) / sigma^2 without a product, dSigma_tau^2 = I
 *   gives M = L^-1 L^-T.  (A location met twice makes two rows of Sigma equal:
 *   no factor, so zero distances are on the diagonal only.)  2.67 N^3 flops,
 *   4 N^3 with the nugget, where S = Sigma^-1 and full products G_j = S D_j
 *   took 6.67 N^3, and 16 or 24 bytes per element of workspace for 44: device
 *   time with / without the nugget at N = 4000 11.1 / 8.3 ms (15.6 / 15.5),
 *   8000 72 / 51 (113), 16000 511 / 349 (823); DMMA bound.  Error of F
 *   relative to sqrt(F_jj F_kk) against an extended-precision evaluation on the
 *   same Sigma, 42 fields of N = 400 to 4000: 5.3e-14 rms, 1.7e-13 at most
 *   (8.3e-13 and 2.0e-12).  The derivatives
 *   come from core_dcmg_matern_dsigma_square / _dbeta / _dnu
 *   (exageostat_exact/cpu_core/compute/core_zcmg.c:315-488; the nu derivative
 *   of K_nu is exact instead of the reference's 1e-9 forward difference,
 *   core_zcmg.c:228-235).
 *
 * MLOE / MMOM (EXAGEOSTAT_dmle_mloe_mmom_Tile, MLE_dexact.c:1109-1434, with
 * the per-point accumulation of CORE_dmloe_mmom_starpu,
 * exageostat_exact/runtime/starpu/codelets/codelet_zmloe_mmom.c:22-60):
 *   the reference loops over the missing points, each with four
 *   triangular solves and a triangular multiply of one vector against the
 *   full factors.  Here all missing points are right-hand sides of the same
 *   tile solves (an "R layout" matrix: one row per missing point, tile (R, K)
 *   at slot K mt + R), so the work runs on the FP64 tensor cores:
 *     A = L_a^-1 k_a,  U = L_a^-1 k_t,  T = L_t^-1 k_t      (forward solves)
 *     W = L_a^-T A = K_a^-1 k_a        (a forward solve with L_a reversed)
 *     V = L_t^T W                      (triangular product with L_t's tiles transposed in place)
 *   and per missing point (one reduction kernel)
 *     expr1 = U.A,  expr2 = sigma_t^2 - 2 expr1 + V.V,
 *     expr3 = sigma_t^2 - T.T,  expr4 = sigma_a^2 - A.A,
 *     loe = expr2 / expr3 - 1,  mom = expr4 / expr2 - 1   (-1 on a zero denominator).
 */
#include <math.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include <vector>

#include "../../include/exageostat_b200.h"
#include "kbessel.cuh"
#include "xg_common.cuh"
#include "xg_engine.h"
#include "xg_kernels.h"
#include "xg_matern.cuh"

#define XG_AS_ROWS 8

/* ------------------------------------------------------------------------- */
/* MLOE / MMOM kernels                                                       */
/* ------------------------------------------------------------------------- */

/* Cross-covariance k(obs o, miss m) in R layout: row m, column o of tile
 * (m / ts, o / ts) at slot (o / ts) mt + m / ts; zero outside nmiss x nobs.
 * One CTA: XG_AS_ROWS rows of one tile. */
__global__ void __launch_bounds__(256) xg_cross_gen_r_kernel(double *__restrict__ D, int mt, int ts,
                                                             const double *__restrict__ xm,
                                                             const double *__restrict__ ym, int nmiss,
                                                             const double *__restrict__ xo,
                                                             const double *__restrict__ yo, int nobs,
                                                             XgMaternParams p, int metric)
{
    const int strips = ts / XG_AS_ROWS;
    const long long slot = blockIdx.x / strips;
    const int strip = blockIdx.x % strips;
    const int K = (int)(slot / mt), R = (int)(slot % mt);
    double *tile = D + slot * (long long)ts * ts;
    for (int rr = 0; rr < XG_AS_ROWS; ++rr) {
        const int r = strip * XG_AS_ROWS + rr;
        const int m = R * ts + r;
        const bool mok = m < nmiss;
        const double x2 = mok ? xm[m] : 0.0, y2 = mok ? ym[m] : 0.0;
        for (int c = threadIdx.x; c < ts; c += blockDim.x) {
            const int o = K * ts + c;
            double v = 0.0;
            if (mok && o < nobs) v = xg_matern_value(xg_distance(xo[o], yo[o], x2, y2, metric), p);
            tile[(long long)r * ts + c] = v;
        }
    }
}

void xg_launch_cross_gen_r(double *D, int mt, int nt, int ts, const double *xm, const double *ym, int nmiss,
                           const double *xo, const double *yo, int nobs, const XgMaternParams &p, int metric,
                           cudaStream_t st)
{
    const long long blocks = (long long)mt * nt * (ts / XG_AS_ROWS);
    xg_cross_gen_r_kernel<<<(unsigned)blocks, 256, 0, st>>>(D, mt, ts, xm, ym, nmiss, xo, yo, nobs, p, metric);
}

/* Every tile of a packed store transposed in place: one CTA swaps the 32 x 32
 * blocks (a, b) and (b, a), a >= b, of one tile. */
__global__ void __launch_bounds__(256) xg_tile_transpose_kernel(double *__restrict__ D, int ts, int npairs)
{
    __shared__ double s1[32][33], s2[32][33];
    const long long t = blockIdx.x / npairs;
    int a, b;
    xg_pair_decode(blockIdx.x % npairs, &a, &b);
    double *tile = D + t * (long long)ts * ts;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int i = ty; i < 32; i += 8) {
        s1[i][tx] = tile[(long long)(a * 32 + i) * ts + b * 32 + tx];
        s2[i][tx] = tile[(long long)(b * 32 + i) * ts + a * 32 + tx];
    }
    __syncthreads();
    for (int i = ty; i < 32; i += 8) {
        tile[(long long)(a * 32 + i) * ts + b * 32 + tx] = s2[tx][i];
        tile[(long long)(b * 32 + i) * ts + a * 32 + tx] = s1[tx][i];
    }
}

void xg_launch_tile_transpose(double *D, long long ntiles, int ts, cudaStream_t st)
{
    const int nb = ts / 32, npairs = nb * (nb + 1) / 2;
    xg_tile_transpose_kernel<<<(unsigned)(ntiles * npairs), 256, 0, st>>>(D, ts, npairs);
}

/* A lower-tile factor L of order P = nt ts and its inverted diagonal blocks
 * replaced by J L^T J, J the reversal of 0 .. P - 1, which is lower triangular
 * again: element (r, c) moves to (P - 1 - c, P - 1 - r).  One CTA swaps two
 * 32 x 32 blocks; the diagonal blocks from row `used` on are the identity, and
 * so are their inverses, which the factorisation leaves unwritten.  The
 * backward solve becomes a forward one, in the same dataflow launch: all the
 * solves and products of MLOE / MMOM in ms, before / after, 1000 + 100
 * locations 1.00 / 0.64, 4000 + 400 4.13 / 2.81, 20000 + 1000 76.1 / 66.3 (a
 * launch per tile column with 32-row strips by serial substitution, 110 us
 * each, took the difference). */
__device__ __forceinline__ void xg_swap_reversed(double *p, double *q, int ld, bool unit_p, bool unit_q,
                                                 double (*s1)[33], double (*s2)[33])
{
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int i = ty; i < 32; i += 8) {
        const double one = i == tx ? 1.0 : 0.0;
        s1[i][tx] = unit_p ? one : p[(long long)i * ld + tx];
        s2[i][tx] = unit_q ? one : q[(long long)i * ld + tx];
    }
    __syncthreads();
    for (int i = ty; i < 32; i += 8) {
        if (p != q) p[(long long)i * ld + tx] = s2[31 - tx][31 - i];
        q[(long long)i * ld + tx] = s1[31 - tx][31 - i];
    }
}

__global__ void __launch_bounds__(256) xg_reverse_factor_kernel(double *__restrict__ L, const int2 *__restrict__ ij,
                                                                double *__restrict__ dinv, long long ntiles, int nt,
                                                                int ts, int used)
{
    __shared__ double s1[32][33], s2[32][33];
    const int nb = ts / 32;
    const long long t = blockIdx.x / (nb * nb);
    if (t < ntiles) {
        const int a = (int)(blockIdx.x % (nb * nb)) / nb, b = (int)(blockIdx.x % (nb * nb)) % nb;
        const int2 at = ij[t];
        const long long u = xg_tile_index(nt - 1 - at.y, nt - 1 - at.x, nt);
        const int ua = nb - 1 - b, ub = nb - 1 - a;
        if (u < t || (u == t && (ua < a || (ua == a && ub < b)))) return; /* the partner's CTA does it */
        xg_swap_reversed(L + (t * ts + a * 32) * ts + b * 32, L + (u * ts + ua * 32) * ts + ub * 32, ts, false,
                         false, s1, s2);
    } else { /* the inverted diagonal blocks */
        const long long n = (long long)nt * nb, e = n - 1 - (blockIdx.x - ntiles * nb * nb), f = n - 1 - e;
        if (e < f) return;
        xg_swap_reversed(dinv + e * 1024, dinv + f * 1024, 32, 32 * e >= used, 32 * f >= used, s1, s2);
    }
}

void xg_launch_reverse_factor(double *L, const int2 *ij, double *dinv, int nt, int ts, int used, cudaStream_t st)
{
    const long long ntiles = xg_num_lower_tiles(nt), nb = ts / 32;
    xg_reverse_factor_kernel<<<(unsigned)(ntiles * nb * nb + nt * nb), 256, 0, st>>>(L, ij, dinv, ntiles, nt, ts, used);
}

/* dst(:, c) = src(:, P - 1 - c) for an R-layout matrix of mt nt tiles */
__global__ void __launch_bounds__(256) xg_reverse_columns_kernel(double *__restrict__ dst,
                                                                 const double *__restrict__ src, int mt, int nt, int ts)
{
    const long long row = blockIdx.x; /* of dst's store: tile slot ts + row in the tile */
    const long long slot = row / ts;
    const int K = (int)(slot / mt), R = (int)(slot - (long long)K * mt);
    const double *from = src + (((long long)(nt - 1 - K) * mt + R) * ts + row % ts) * ts;
    for (int c = threadIdx.x; c < ts; c += blockDim.x) dst[row * ts + c] = from[ts - 1 - c];
}

void xg_launch_reverse_columns(double *dst, const double *src, int mt, int nt, int ts, cudaStream_t st)
{
    xg_reverse_columns_kernel<<<(unsigned)((long long)mt * nt * ts), 256, 0, st>>>(dst, src, mt, nt, ts);
}

/* One CTA per missing point m: the four row sums over its R-layout row in A,
 * U, T, V, combined into terms[6 m ..] = expr1, expr2, expr3, expr4, loe, mom. */
__global__ void __launch_bounds__(256) xg_mloe_terms_kernel(const double *__restrict__ A, const double *__restrict__ U,
                                                            const double *__restrict__ T, const double *__restrict__ V,
                                                            int mt, int nt, int ts, double sigma2_t, double sigma2_a,
                                                            double *__restrict__ terms)
{
    __shared__ double red[4][8];
    const int m = blockIdx.x;
    const int R = m / ts, r = m % ts;
    double s[4] = {0.0, 0.0, 0.0, 0.0}; /* A.A, U.A, T.T, V.V */
    for (int K = 0; K < nt; ++K) {
        const long long off = (((long long)K * mt + R) * ts + r) * ts;
        for (int c = threadIdx.x; c < ts; c += blockDim.x) {
            const double a = A[off + c], u = U[off + c], t = T[off + c], v = V[off + c];
            s[0] += a * a;
            s[1] += u * a;
            s[2] += t * t;
            s[3] += v * v;
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        double v = s[q];
        for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        if (lane == 0) red[q][warp] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double tot[4];
        for (int q = 0; q < 4; ++q) {
            double v = 0.0;
            for (int w = 0; w < 8; ++w) v += red[q][w];
            tot[q] = v;
        }
        /* MLE_dexact.c:1371-1375: expr1 <- alpha_t - 2 expr1, expr2 <- expr1 + expr2,
         * expr3 <- alpha_t - expr3, expr4 <- alpha_a - expr4 */
        const double e1 = tot[1];
        const double e2 = (sigma2_t - 2.0 * e1) + tot[3];
        const double e3 = sigma2_t - tot[2];
        const double e4 = sigma2_a - tot[0];
        double *o = terms + 6 * (long long)m;
        o[0] = e1;
        o[1] = e2;
        o[2] = e3;
        o[3] = e4;
        o[4] = e3 == 0.0 ? -1.0 : e2 / e3 - 1.0; /* codelet_zmloe_mmom.c:48-53 */
        o[5] = e2 == 0.0 ? -1.0 : e4 / e2 - 1.0; /* :55-60 */
    }
}

void xg_launch_mloe_terms(const double *A, const double *U, const double *T, const double *V, int mt, int nt, int ts,
                          int nmiss, double sigma2_t, double sigma2_a, double *terms, cudaStream_t st)
{
    xg_mloe_terms_kernel<<<nmiss, 256, 0, st>>>(A, U, T, V, mt, nt, ts, sigma2_t, sigma2_a, terms);
}

/* ------------------------------------------------------------------------- */
/* Fisher kernels                                                            */
/* ------------------------------------------------------------------------- */

/* Y^T into the lower half of the square R-layout matrices Y, Y + full, ..:
 * the 32 x 32 block (a, b), a >= b, becomes the transpose of (b, a). */
__global__ void __launch_bounds__(256) xg_lower_transpose_kernel(double *__restrict__ Y, int nt, int ts)
{
    __shared__ double s[32][33];
    const int nb = ts / 32;
    int a, b;
    xg_pair_decode(blockIdx.x, &a, &b);
    double *F = Y + blockIdx.y * (long long)nt * nt * ts * ts;
    const double *src = F + (((long long)(a / nb) * nt + b / nb) * ts + b % nb * 32) * ts + a % nb * 32;
    double *dst = F + (((long long)(b / nb) * nt + a / nb) * ts + a % nb * 32) * ts + b % nb * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int i = ty; i < 32; i += 8) s[i][tx] = src[(long long)i * ts + tx];
    __syncthreads();
    for (int i = ty; i < 32; i += 8) dst[(long long)i * ts + tx] = s[tx][i];
}

void xg_launch_lower_transpose(double *Y, int nsys, int nt, int ts, cudaStream_t st)
{
    const long long nb = (long long)nt * (ts / 32);
    xg_lower_transpose_kernel<<<dim3((unsigned)(nb * (nb + 1) / 2), nsys), 256, 0, st>>>(Y, nt, ts);
}

/* dSigma/dtheta_which (1 beta, 2 nu, 3 tau^2) into a square R-layout matrix,
 * zero outside N x N and, for beta and nu, at zero distance
 * (core_zcmg.c:394-395, 471-472). */
__global__ void __launch_bounds__(256) xg_dsigma_full_kernel(double *__restrict__ D, int nt, int ts,
                                                             const double *__restrict__ x,
                                                             const double *__restrict__ y, int N, XgMaternParams p,
                                                             double dlogcon, int metric, int which)
{
    const int strips = ts / XG_AS_ROWS;
    const long long slot = blockIdx.x / strips;
    const int strip = blockIdx.x % strips;
    const int B = (int)(slot / nt), A = (int)(slot % nt);
    double *tile = D + slot * (long long)ts * ts;
    for (int rr = 0; rr < XG_AS_ROWS; ++rr) {
        const int r = strip * XG_AS_ROWS + rr;
        const int ga = A * ts + r;
        const bool rok = ga < N;
        const double x1 = rok ? x[ga] : 0.0, y1 = rok ? y[ga] : 0.0;
        for (int c = threadIdx.x; c < ts; c += blockDim.x) {
            const int gb = B * ts + c;
            double v = 0.0;
            if (rok && gb < N) {
                if (which == 3) {
                    v = ga == gb ? 1.0 : 0.0;
                } else {
                    const double rd = xg_distance(x1, y1, x[gb], y[gb], metric) / p.beta;
                    if (rd != 0.0) {
                        double m, ds, db, dn;
                        xg_matern_grad(rd, p.nu, p.con, p.sigma2, p.beta, dlogcon, &m, &ds, &db, &dn);
                        v = which == 1 ? db : dn;
                    }
                }
            }
            tile[(long long)r * ts + c] = v;
        }
    }
}

void xg_launch_dsigma_full(double *D, int nt, int ts, const double *x, const double *y, int N,
                           const XgMaternParams &p, double dlogcon, int metric, int which, double *tab,
                           cudaStream_t st)
{
    if (which < 3 && tab && xg_tab_covers(p, N)) {
        if (which == 1) xg_launch_grad_tables(p, dlogcon, tab, st); /* the call for 2 follows on the stream */
        xg_launch_dsigma_full_tab(D, nt, ts, x, y, N, p, dlogcon, metric, which, tab, st);
        return;
    }
    const long long blocks = (long long)nt * nt * (ts / XG_AS_ROWS);
    xg_dsigma_full_kernel<<<(unsigned)blocks, 256, 0, st>>>(D, nt, ts, x, y, N, p, dlogcon, metric, which);
}

/* part[10 blockIdx.x + q] for the pairs q = (j, k), j <= k < 4, in row order
 * (pairs with k >= np stay zero): sum over a, b < N of W_j[a, b] W_k[a, b],
 * from the lower halves of W_1, W_2 (, M) at W, W + full (, W + 2 full). */
__global__ void __launch_bounds__(256) xg_fisher_trace_kernel(const double *__restrict__ W, int np, int nt, int ts,
                                                              int N, long long units, double inv_sigma2, double nugget,
                                                              double *__restrict__ part)
{
    __shared__ double red[10][8];
    const int nb = ts / XG_DAG_BLOCK;
    const long long full = (long long)nt * nt * ts * ts;
    double acc[10];
#pragma unroll
    for (int q = 0; q < 10; ++q) acc[q] = 0.0;
    for (long long u = blockIdx.x; u < units; u += gridDim.x) { /* 32 rows of a lower 128-block */
        int I, J;
        xg_pair_decode(u / 4, &I, &J);
        const int c = 2 * (threadIdx.x & 63), gb = J * XG_DAG_BLOCK + c;
        for (int i = 0; i < 8; ++i) {
            const int r = (int)(u % 4) * 32 + 4 * i + (int)(threadIdx.x >> 6), ga = I * XG_DAG_BLOCK + r;
            if (ga >= N || gb > ga) continue;
            const double *at = W + (((long long)(J / nb) * nt + I / nb) * ts + I % nb * XG_DAG_BLOCK + r) * ts +
                               J % nb * XG_DAG_BLOCK + c;
            double2 w[3];
#pragma unroll
            for (int m = 0; m < 3; ++m)
                w[m] = m < np - 1 ? *(const double2 *)(at + m * full) : make_double2(0.0, 0.0);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (gb + h > ga) continue;
                const double d = ga == gb + h ? 1.0 : 0.0, f = 2.0 - d; /* the mirror counts too */
                double P[4];
#pragma unroll
                for (int m = 0; m < 3; ++m) P[m + 1] = h ? w[m].y : w[m].x;
                P[0] = (d - nugget * P[3]) * inv_sigma2;
                int q = 0;
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int k = j; k < 4; ++k, ++q) acc[q] += f * P[j] * P[k];
            }
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < 10; ++q) {
        double v = acc[q];
        for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        if (lane == 0) red[q][warp] = v;
    }
    __syncthreads();
    if (threadIdx.x < 10) {
        double v = 0.0;
        for (int w = 0; w < 8; ++w) v += red[threadIdx.x][w];
        part[10 * (long long)blockIdx.x + threadIdx.x] = v;
    }
}

void xg_launch_fisher_trace(const double *W, int np, int nt, int ts, int N, double sigma2, double nugget, double *part,
                            int nctas, cudaStream_t st)
{
    const long long units = 4 * xg_num_lower_tiles((N + XG_DAG_BLOCK - 1) / XG_DAG_BLOCK);
    xg_fisher_trace_kernel<<<nctas, 256, 0, st>>>(W, np, nt, ts, N, units, 1.0 / sigma2, nugget, part);
}

/* ------------------------------------------------------------------------- */
/* host: Fisher information                                                  */
/* ------------------------------------------------------------------------- */

#define XG_ACU(call)                                                                                                   \
    do {                                                                                                               \
        cudaError_t _e = (call);                                                                                       \
        if (_e != cudaSuccess) return xg_fail(XG_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(_e));                   \
    } while (0)

static int xg_status_error(const int sv[2], const char *what)
{
    if (sv[0] & XG_ST_NOT_SPD) return xg_fail(XG_ERR_NOT_SPD, "%s is not positive definite (pivot %d)", what, sv[1]);
    if (sv[0] & XG_ST_TIMEOUT) return xg_fail(XG_ERR_TIMEOUT, "a device pipeline wait timed out");
    return xg_fail(XG_ERR_CUDA, "device status word 0x%x", sv[0]);
}

/* n x n SPD inverse as EXAGEOSTAT_Fisher_Tile does it (MLE_dexact.c:1893-1916):
 * A = L L^T, then X = L^-T (L^-1 I).  A and inv row-major (A symmetric). */
int xg_small_spd_inverse(int n, const double *A, double *inv)
{
    double L[16] = {0};
    for (int j = 0; j < n; ++j) {
        double d = A[j * n + j];
        for (int k = 0; k < j; ++k) d -= L[j * n + k] * L[j * n + k];
        if (!(d > 0.0)) return xg_fail(XG_ERR_NOT_SPD, "the Fisher matrix is not positive definite");
        L[j * n + j] = sqrt(d);
        for (int i = j + 1; i < n; ++i) {
            double s = A[i * n + j];
            for (int k = 0; k < j; ++k) s -= L[i * n + k] * L[j * n + k];
            L[i * n + j] = s / L[j * n + j];
        }
    }
    for (int c = 0; c < n; ++c) {
        double y[4];
        for (int i = 0; i < n; ++i) { /* L y = e_c */
            double s = i == c ? 1.0 : 0.0;
            for (int k = 0; k < i; ++k) s -= L[i * n + k] * y[k];
            y[i] = s / L[i * n + i];
        }
        for (int i = n - 1; i >= 0; --i) { /* L^T x = y */
            double s = y[i];
            for (int k = i + 1; k < n; ++k) s -= L[k * n + i] * inv[k * n + c];
            inv[i * n + c] = s / L[i * n + i];
        }
    }
    return XG_OK;
}

/* Fisher information of the field's locations at theta: kernel 0 gives the
 * 3 x 3 matrix of (sigma^2, beta, nu), kernel 1 the 4 x 4 one with tau^2.
 * F row-major; seconds = device time of the whole computation.  The field's
 * covariance store is overwritten (the next evaluation regenerates it). */
int xg_field_fisher(XgField *f, const double *theta, int kernel, double *F, double *seconds)
{
    if (xg_bivariate(kernel) || xg_bivariate(f->kernel))
        return xg_fail(XG_ERR_UNSUPPORTED, "the Fisher matrix of a bivariate field");
    int rc = xg_check_theta(theta, kernel);
    if (rc) return rc;
    const int nt = f->C.nt, ts = f->C.ts, N = f->N;
    const int np = kernel == 1 ? 4 : 3, nsys = np - 1;
    const int nb = (N + XG_DAG_BLOCK - 1) / XG_DAG_BLOCK;
    const size_t full = (size_t)nt * nt * ts * ts;
    const size_t words = 2 + (size_t)nsys * nb * nb; /* next task, abort, block flags */
    const int nctas = g_xg.sm_count * 8;
    double *Y = nullptr, *part = nullptr;
    int *w = nullptr;
    const XgPart parts[] = {{&Y, nsys * full}, {&part, 10 * (size_t)nctas}, {&w, words}};
    if (xg_alloc_parts(parts, 3) != cudaSuccess)
        return xg_fail(XG_ERR_NO_MEMORY, "Fisher workspace: %.2f GB", nsys * full * sizeof(double) / 1e9);
    XgI8Use use(f->C, xg_params(theta, kernel));
    std::vector<double> hp(10 * (size_t)nctas);
    int sv[2] = {0, 0};
    XgRowsMaps maps = {};
    XgRows R = {};
    for (int k = 0; k < nsys && !rc; ++k) {
        rc = xg_encode_tiles(&maps.y[k], Y + k * full, (long long)nt * nt, ts);
        maps.l[k] = f->C.map;
        R.y[k] = Y + k * full;
        R.dinv[k] = f->C.dinv;
    }
    R.ts = ts;
    R.nsys = nsys;
    R.one.nt = R.one.mt = nt;
    R.one.nb = R.one.mr = nb;
    R.sys_flags = (long long)nb * nb;
    R.next = (unsigned *)w;
    R.abort = w + 1;
    R.flags = w + 2;
    R.status = f->status;
    if (!rc) {
        cudaStream_t st = g_xg.stream;
        XgTileArgs T{f->C.d, ts, nt};
        const XgMaternParams p = xg_params(theta, kernel);
        const double dlogcon = -(log(2.0) + xg_digamma(theta[2]));
        cudaMemsetAsync(f->status, 0, 2 * sizeof(int), st);
        cudaEventRecord(f->ev[0], st);
        /* Sigma (MLE_dexact.c:1824-1825) and its factor (:1830) */
        xg_launch_gen(T, f->C.ij, f->C.ntiles, f->x, f->y, f->x, f->y, N, N, p, f->metric, 1, f->C.tab, st);
        XgFactorStreams fs;
        fs.st = st;
        fs.st_hi = g_xg.stream_hi;
        fs.ev_panel = f->ev_panel;
        fs.ev_upd = f->ev_upd;
        xg_factor_lookahead(f->C, nullptr, f->part, f->status, f->info, fs);
        /* Y_j = dSigma_j L^-T, then the lower half of W_j = L^-1 Y_j */
        for (int k = 0; k < nsys; ++k)
            xg_launch_dsigma_full(Y + k * full, nt, ts, f->x, f->y, N, p, dlogcon, f->metric, k + 1, f->C.tab, st);
        cudaMemsetAsync(w, 0, words * sizeof(int), st);
        R.ntasks = (long long)nsys * nb * nb;
        xg_launch_rows(XG_ROWS_RHS, maps, R, g_xg.sm_count, st);
        xg_launch_lower_transpose(Y, nsys, nt, ts, st);
        cudaMemsetAsync(w, 0, words * sizeof(int), st);
        R.lower = 1;
        R.ntasks = nsys * xg_num_lower_tiles(nb);
        xg_launch_rows(XG_ROWS_RHS, maps, R, g_xg.sm_count, st);
        xg_launch_fisher_trace(Y, np, nt, ts, N, p.sigma2, p.nugget, part, nctas, st);
        cudaEventRecord(f->ev[3], st);
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(hp.data(), part, hp.size() * sizeof(double), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(sv, f->status, sizeof sv, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) rc = xg_fail(XG_ERR_CUDA, "Fisher: %s", cudaGetErrorString(e));
        if (!rc && seconds) {
            float ms = 0;
            cudaEventElapsedTime(&ms, f->ev[0], f->ev[3]);
            *seconds = ms * 1e-3;
        }
    }
    cudaFree(Y);
    if (rc) return rc;
    if (sv[0]) return xg_status_error(sv, "the covariance");
    int q = 0;
    for (int j = 0; j < 4; ++j)
        for (int k = j; k < 4; ++k, ++q) {
            if (k >= np) continue;
            double s = 0.0;
            for (int b = 0; b < nctas; ++b) s += hp[10 * (size_t)b + q];
            F[j * np + k] = F[k * np + j] = 0.5 * s;
        }
    return XG_OK;
}

/* ------------------------------------------------------------------------- */
/* host: MLOE / MMOM                                                         */
/* ------------------------------------------------------------------------- */

void xg_assess_destroy(XgAssess *q)
{
    if (!q) return;
    xg_tm_free(q->Ca);
    xg_tm_free(q->Ct);
    cudaFree(q->R[0]);
    for (int i = 0; i < 4; ++i)
        if (q->ev[i]) cudaEventDestroy(q->ev[i]);
    if (q->ev_panel) cudaEventDestroy(q->ev_panel);
    if (q->ev_upd) cudaEventDestroy(q->ev_upd);
    delete q;
}

int xg_assess_create(XgAssess **out, int nmiss, int nobs, int ts)
{
    *out = nullptr;
    int rc = xg_context_require();
    if (rc) return rc;
    if (nmiss <= 0 || nobs <= 0) return xg_fail(XG_ERR_BAD_ARGUMENT, "nZmiss = %d, nZobs = %d", nmiss, nobs);
    XgAssess *q = new XgAssess();
    q->nmiss = nmiss;
    q->nobs = nobs;
    q->ts = xg_choose_ts(nobs, ts);
    rc = xg_tm_alloc(q->Ca, nobs, q->ts);
    if (!rc) rc = xg_tm_alloc(q->Ct, nobs, q->ts);
    q->nt = q->Ca.nt;
    q->mt = (nmiss + q->ts - 1) / q->ts;
    const long long rtiles = (long long)q->mt * q->nt;
    const size_t Np = (size_t)q->nt * q->ts, rsize = (size_t)rtiles * q->ts * q->ts;
    /* three forward solves, or the backward one with the padding's blocks */
    const long long nb = (nobs + XG_DAG_BLOCK - 1) / XG_DAG_BLOCK, nbp = (long long)Np / XG_DAG_BLOCK;
    const long long flags = (3 * nb > nbp ? 3 * nb : nbp) * ((nmiss + XG_DAG_BLOCK - 1) / XG_DAG_BLOCK);
    if (!rc) {
        const XgPart parts[] = {{&q->R[0], rsize}, {&q->R[1], rsize}, {&q->R[2], rsize}, {&q->R[3], rsize},
                                {&q->R[4], rsize}, {&q->xo, Np}, {&q->yo, Np}, {&q->xm, (size_t)nmiss},
                                {&q->ym, (size_t)nmiss}, {&q->terms, 6 * (size_t)nmiss},
                                {&q->part, 4 * Np / XG_DAG_BLOCK}, {&q->status, 2}, {&q->words, (size_t)(2 + flags)}};
        cudaError_t e = xg_alloc_parts(parts, 13);
        /* on the stream that fills them: the default stream does not wait for it, nor it for that */
        if (e == cudaSuccess)
            e = cudaMemsetAsync(q->R[0], 0, (char *)(q->words + 2 + flags) - (char *)q->R[0], g_xg.stream);
        if (e != cudaSuccess)
            rc = xg_fail(XG_ERR_NO_MEMORY, "MLOE / MMOM workspace (%.2f GB): %s", 5.0 * rsize * sizeof(double) / 1e9,
                         cudaGetErrorString(e));
    }
    for (int i = 0; i < 5 && !rc; ++i) rc = xg_encode_tiles(&q->mR[i], q->R[i], rtiles, q->ts);
    for (int i = 0; i < 4 && !rc; ++i)
        if (cudaEventCreate(&q->ev[i]) != cudaSuccess) rc = xg_fail(XG_ERR_CUDA, "events");
    if (!rc && (cudaEventCreateWithFlags(&q->ev_panel, cudaEventDisableTiming) != cudaSuccess ||
                cudaEventCreateWithFlags(&q->ev_upd, cudaEventDisableTiming) != cudaSuccess))
        rc = xg_fail(XG_ERR_CUDA, "lookahead events");
    if (rc) {
        xg_assess_destroy(q);
        return rc;
    }
    *out = q;
    return XG_OK;
}

/* mloe / mmom (means over the missing points), terms (6 per point, optional)
 * and times[4] = generation, the two factorisations, the solves and
 * reductions, total (seconds, CUDA events). */
int xg_assess_run(XgAssess *q, const double *truth, const double *est, int kernel, int metric, const double *xm,
                  const double *ym, const double *xo, const double *yo, double *mloe, double *mmom, double *terms,
                  double *times)
{
    int rc = xg_check_theta(truth, kernel);
    if (!rc) rc = xg_check_theta(est, kernel);
    if (rc) return rc;
    cudaStream_t st = g_xg.stream;
    const int nmiss = q->nmiss, nobs = q->nobs, nt = q->nt, mt = q->mt, ts = q->ts;
    const XgMaternParams pt = xg_params(truth, kernel), pa = xg_params(est, kernel);
    XgI8Use use_a(q->Ca, pa), use_t(q->Ct, pt);
    double *RA = q->R[0], *RU = q->R[1], *RT = q->R[2], *RW = q->R[3], *RV = q->R[4];
    const size_t rbytes = (size_t)mt * nt * ts * ts * sizeof(double);
    XG_ACU(cudaMemsetAsync(q->status, 0, 2 * sizeof(int), st));
    XG_ACU(cudaMemcpyAsync(q->xo, xo, nobs * sizeof(double), cudaMemcpyHostToDevice, st));
    XG_ACU(cudaMemcpyAsync(q->yo, yo, nobs * sizeof(double), cudaMemcpyHostToDevice, st));
    XG_ACU(cudaMemcpyAsync(q->xm, xm, nmiss * sizeof(double), cudaMemcpyHostToDevice, st));
    XG_ACU(cudaMemcpyAsync(q->ym, ym, nmiss * sizeof(double), cudaMemcpyHostToDevice, st));
    XG_ACU(cudaEventRecord(q->ev[0], st));
    /* K_a = Sigma(obs, obs; estimated), K_t (truth) (MLE_dexact.c:1239-1245),
     * k_a and k_t for every missing point at once (:1283-1286) */
    XgTileArgs Ta{q->Ca.d, ts, nt}, Tt{q->Ct.d, ts, nt};
    xg_launch_gen(Ta, q->Ca.ij, q->Ca.ntiles, q->xo, q->yo, q->xo, q->yo, nobs, nobs, pa, metric, 1, q->Ca.tab, st);
    xg_launch_gen(Tt, q->Ct.ij, q->Ct.ntiles, q->xo, q->yo, q->xo, q->yo, nobs, nobs, pt, metric, 1, q->Ct.tab, st);
    xg_launch_cross_gen_r(RA, mt, nt, ts, q->xm, q->ym, nmiss, q->xo, q->yo, nobs, pa, metric, st);
    xg_launch_cross_gen_r(RU, mt, nt, ts, q->xm, q->ym, nmiss, q->xo, q->yo, nobs, pt, metric, st);
    XG_ACU(cudaMemcpyAsync(RT, RU, rbytes, cudaMemcpyDeviceToDevice, st));
    XG_ACU(cudaEventRecord(q->ev[1], st));
    /* the two factorisations (:1252, :1261) */
    XgFactorStreams fs;
    fs.st = st;
    fs.st_hi = g_xg.stream_hi;
    fs.ev_panel = q->ev_panel;
    fs.ev_upd = q->ev_upd;
    xg_factor_two(q->Ca, q->Ct, q->part, q->part + 2 * (size_t)nt * ts / XG_DAG_BLOCK, q->status, q->status + 1, fs);
    XG_ACU(cudaEventRecord(q->ev[2], st));
    /* the per-point solves (:1300-1364) for all points */
    {
        /* A = L_a^-1 k_a, U = L_a^-1 k_t, T = L_t^-1 k_t */
        const XgTileMatrix *L[3] = {&q->Ca, &q->Ca, &q->Ct};
        XgRowsMaps maps;
        XgRows G = {};
        for (int i = 0; i < 3; ++i) {
            maps.y[i] = q->mR[i];
            maps.l[i] = L[i]->map;
            G.y[i] = q->R[i];
            G.dinv[i] = L[i]->dinv;
        }
        G.ts = ts;
        G.nsys = 3;
        G.one.nt = nt;
        G.one.nb = (nobs + XG_DAG_BLOCK - 1) / XG_DAG_BLOCK;
        G.one.mt = mt;
        G.one.mr = (nmiss + XG_DAG_BLOCK - 1) / XG_DAG_BLOCK;
        G.sys_flags = (long long)G.one.nb * G.one.mr;
        G.ntasks = 3 * G.sys_flags;
        G.next = (unsigned *)q->words;
        G.abort = q->words + 1;
        G.flags = q->words + 2;
        G.status = q->status;
        XG_ACU(cudaMemsetAsync(q->words, 0, sizeof(int) * (size_t)(2 + 3 * G.sys_flags), st));
        xg_launch_rows(XG_ROWS_RHS, maps, G, g_xg.sm_count, st);
    }
    /* W = L_a^-T A: with J the reversal, (W J) (J L_a J) = A J is a forward solve with J L_a^T J */
    xg_launch_reverse_factor(q->Ca.d, q->Ca.ij, q->Ca.dinv, nt, ts, (nobs + XG_DAG_BLOCK - 1) / XG_DAG_BLOCK * XG_DAG_BLOCK,
                             st);
    xg_launch_reverse_columns(RV, RA, mt, nt, ts, st);
    {
        XgRowsMaps maps;
        XgRows G = {};
        maps.y[0] = q->mR[4];
        maps.l[0] = q->Ca.map;
        G.y[0] = RV;
        G.dinv[0] = q->Ca.dinv;
        G.ts = ts;
        G.nsys = 1;
        G.one.nt = nt;
        G.one.nb = nt * (ts / XG_DAG_BLOCK); /* the padding comes first */
        G.one.mt = mt;
        G.one.mr = (nmiss + XG_DAG_BLOCK - 1) / XG_DAG_BLOCK;
        G.ntasks = G.sys_flags = (long long)G.one.nb * G.one.mr;
        G.next = (unsigned *)q->words;
        G.abort = q->words + 1;
        G.flags = q->words + 2;
        G.status = q->status;
        XG_ACU(cudaMemsetAsync(q->words, 0, sizeof(int) * (size_t)(2 + G.sys_flags), st));
        xg_launch_rows(XG_ROWS_RHS, maps, G, g_xg.sm_count, st);
    }
    xg_launch_reverse_columns(RW, RV, mt, nt, ts, st);
    xg_launch_tile_transpose(q->Ct.d, q->Ct.ntiles, ts, st);
    xg_launch_rhs_tri_product(q->mR[3], q->Ct.map, RV, mt, nt, ts, q->status, st); /* V = L_t^T W */
    xg_launch_mloe_terms(RA, RU, RT, RV, mt, nt, ts, nmiss, truth[0], est[0], q->terms, st);
    XG_ACU(cudaEventRecord(q->ev[3], st));
    XG_ACU(cudaGetLastError());
    std::vector<double> h(6 * (size_t)nmiss);
    int sv[2];
    XG_ACU(cudaMemcpyAsync(h.data(), q->terms, h.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
    XG_ACU(cudaMemcpyAsync(sv, q->status, sizeof sv, cudaMemcpyDeviceToHost, st));
    XG_ACU(cudaStreamSynchronize(st));
    if (sv[0]) return xg_status_error(sv, "K_a or K_t");
    double sl = 0.0, sm = 0.0;
    for (int m = 0; m < nmiss; ++m) {
        sl += h[6 * (size_t)m + 4];
        sm += h[6 * (size_t)m + 5];
    }
    *mloe = sl / nmiss;
    *mmom = sm / nmiss;
    if (terms) memcpy(terms, h.data(), h.size() * sizeof(double));
    if (times) {
        float a = 0, b = 0, c = 0;
        cudaEventElapsedTime(&a, q->ev[0], q->ev[1]);
        cudaEventElapsedTime(&b, q->ev[1], q->ev[2]);
        cudaEventElapsedTime(&c, q->ev[2], q->ev[3]);
        times[0] = a * 1e-3;
        times[1] = b * 1e-3;
        times[2] = c * 1e-3;
        times[3] = (a + b + c) * 1e-3;
    }
    return XG_OK;
}
