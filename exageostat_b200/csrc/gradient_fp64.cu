/*
 * Gradient of the exact Matern log-likelihood (FP64), on sm_100a.
 *
 *   d loglik / d theta_p = 1/2 alpha^T (dSigma/dtheta_p) alpha - 1/2 tr(Sigma^-1 dSigma/dtheta_p)
 *                        = sum_{R,C} W_RC (dSigma/dtheta_p)_RC,   W = (alpha alpha^T - Sigma^-1) / 2,
 * alpha = Sigma^-1 z.  The reference has no gradient (NLopt's derivative-free
 * BOBYQA ignores grad, examples/synthetic_dmle_test.c:140-142); its dSigma/dtheta
 * element kernels (core_dcmg_matern_dsigma_square / _dbeta / _dnu,
 * exageostat_exact/cpu_core/compute/core_zcmg.c:315-488) are the math spec.
 *
 * After the forward factorisation (Sigma = L L^T in the lower tiles):
 *   1. alpha = L^-T (L^-1 z) with the backward solve (solve.cu).
 *   2. X = L^-T, upper triangular (rows_dag.cu; on the INT8 path tile column by
 *      tile column, with the updates of sliced.cu), X_IK stored row-major at packed slot
 *      (K, I) of a second lower-tile buffer, so both GEMM operands stay
 *      K-major for TMA.
 *   3. Sigma^-1 lower = X X^T: S_IJ = sum_{K >= I} X_IK X_JK^T, written over
 *      the factor (rows_dag.cu, or the sliced kernel).
 *   4. One fused pass over the lower tiles of S generates dSigma/dtheta_p on
 *      the fly (never stored) and contracts it with W.
 * Steps 2 and 3 are N^3/3 flops each (TRTRI- and LAUUM-class), so a gradient
 * costs about two extra factorisations.
 */
#include <math.h>
#include <stdint.h>

#include "kbessel.cuh"
#include "xg_common.cuh"
#include "xg_kernels.h"
#include "xg_matern.cuh"

/* ========================================================================== */
/* Triangular product of right-hand sides over 128 x 128 blocks               */
/* ========================================================================== */

#define XG_TG_BM 128
#define XG_TG_BK 16
#define XG_TG_STAGES 4
#define XG_TG_THREADS 256
#define XG_TG_STAGE_BYTES (2 * XG_TG_BM * XG_TG_BK * 8)

/* C(R, I) = sum_{K >= I} A(R, K) B_slot(K, I)^T for "R layout" A and C, an mt x
 * nt grid of tiles whose tile (R, K) sits at slot K * mt + R (right-hand sides
 * stored transposed, one row per right-hand side), and lower-tile packed B. */
__global__ void __launch_bounds__(XG_TG_THREADS, 1)
    xg_tile_gemm_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                        double *__restrict__ Cbase, int nt, int ts, int mt, int *status)
{
    extern __shared__ __align__(1024) unsigned char xg_smem_raw[];
    unsigned char *smem = (unsigned char *)(((uintptr_t)xg_smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t *full = (uint64_t *)(smem + XG_TG_STAGES * XG_TG_STAGE_BYTES);
    uint64_t *empty = full + XG_TG_STAGES;
    const int bpt = ts / XG_TG_BM;
    const long long job = blockIdx.x / (bpt * bpt);
    const int blk = blockIdx.x % (bpt * bpt);
    const int bi = blk / bpt, bj = blk % bpt;
    const int R = (int)(job % mt), I = (int)(job / mt);
    /* the tiles (K, I), K = I .. nt - 1, are consecutive in the packed column I */
    const int c_slot = I * mt + R, b_slot0 = (int)xg_tile_index(I, I, nt);
    if (xg_cta_should_skip(status)) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        for (int s = 0; s < XG_TG_STAGES; ++s) {
            xg_mbar_init(&full[s], 1);
            xg_mbar_init(&empty[s], 8);
        }
        xg_fence_barrier_init();
    }
    __syncthreads();
    const int kper = ts / XG_TG_BK;
    const int KT = (nt - I) * kper;
    auto issue = [&](int q, int s) {
        const int kt = q / kper, kk = (q % kper) * XG_TG_BK;
        const int ya = (c_slot + kt * mt) * ts + bi * XG_TG_BM;
        const int yb = (b_slot0 + kt) * ts + bj * XG_TG_BM;
        unsigned char *sa = smem + s * XG_TG_STAGE_BYTES;
        xg_mbar_arrive_expect_tx(&full[s], XG_TG_STAGE_BYTES);
        xg_tma_load_2d(sa, &mapA, kk, ya, &full[s]);
        xg_tma_load_2d(sa + XG_TG_BM * XG_TG_BK * 8, &mapB, kk, yb, &full[s]);
    };
    int issued = 0;
    if (tid == 0) {
        xg_prefetch_tensormap(&mapA);
        xg_prefetch_tensormap(&mapB);
        for (; issued < XG_TG_STAGES && issued < KT; ++issued) issue(issued, issued);
    }
    const int wm = warp >> 2, wn = warp & 3;
    const int g = lane >> 2, tq = lane & 3;
    double *C = Cbase + (long long)c_slot * ts * ts + (long long)(bi * XG_TG_BM) * ts + bj * XG_TG_BM;
    double acc[4][4][4];
#pragma unroll
    for (int mi = 0; mi < 4; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[mi][ni][e] = 0.0;
    bool ok = true;
    for (int kb = 0; kb < KT; ++kb) {
        const int s = kb % XG_TG_STAGES;
        if (!xg_mbar_wait(&full[s], (kb / XG_TG_STAGES) & 1)) {
            ok = false;
            break;
        }
        const unsigned char *sa = smem + s * XG_TG_STAGE_BYTES;
        const unsigned char *sb = sa + XG_TG_BM * XG_TG_BK * 8;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int chunk = 2 * tq + half;
            double2 b[4];
#pragma unroll
            for (int ni = 0; ni < 4; ++ni) {
                const int r = wn * 32 + ni * 8 + g;
                b[ni] = *(const double2 *)(sb + (r << 7) + ((chunk ^ (r & 7)) << 4));
            }
#pragma unroll
            for (int mi = 0; mi < 4; ++mi) {
                const int r = wm * 64 + mi * 16 + g;
                const double2 a0 = *(const double2 *)(sa + (r << 7) + ((chunk ^ (r & 7)) << 4));
                const double2 a1 = *(const double2 *)(sa + ((r + 8) << 7) + ((chunk ^ ((r + 8) & 7)) << 4));
#pragma unroll
                for (int ni = 0; ni < 4; ++ni) {
                    xg_dmma_16x8x4(acc[mi][ni][0], acc[mi][ni][1], acc[mi][ni][2], acc[mi][ni][3], a0.x, a1.x,
                                   b[ni].x);
                    xg_dmma_16x8x4(acc[mi][ni][0], acc[mi][ni][1], acc[mi][ni][2], acc[mi][ni][3], a0.y, a1.y,
                                   b[ni].y);
                }
            }
        }
        __syncwarp();
        if (lane == 0) xg_mbar_arrive(&empty[s]);
        if (tid == 0 && issued < KT) {
            if (xg_mbar_wait(&empty[s], (kb / XG_TG_STAGES) & 1)) {
                issue(issued, s);
                ++issued;
            } else {
                ok = false;
            }
        }
        __syncwarp();
        if (!ok) break;
    }
    if (!ok) {
        atomicOr(status, XG_ST_TIMEOUT);
        if (tid == 0)
            for (int q = (issued > XG_TG_STAGES ? issued - XG_TG_STAGES : 0); q < issued; ++q)
                xg_mbar_wait(&full[q % XG_TG_STAGES], (q / XG_TG_STAGES) & 1);
        return;
    }
#pragma unroll
    for (int mi = 0; mi < 4; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = wm * 64 + mi * 16 + g + 8 * h;
                const int c = wn * 32 + ni * 8 + 2 * tq;
                *reinterpret_cast<double2 *>(C + (long long)r * ts + c) =
                    make_double2(acc[mi][ni][2 * h], acc[mi][ni][2 * h + 1]);
            }
}

/* zeros the diagonal tiles: the block solves of X = L^-T write only its upper
 * 128-blocks, the digit slicing reads whole tiles */
__global__ void xg_zero_diag_kernel(double *X, int nt, int ts)
{
    double2 *T = reinterpret_cast<double2 *>(X + xg_tile_index((int)blockIdx.y, (int)blockIdx.y, nt) * (long long)ts * ts);
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < ts * ts / 2; e += gridDim.x * blockDim.x)
        T[e] = make_double2(0.0, 0.0);
}

/* ========================================================================== */
/* Fused dSigma/dtheta generation and contraction with W                      */
/* ========================================================================== */

struct XgGradParams {
    double sigma2, beta, nu, nugget, con, dlogcon;
    int kernel; /* 0 Matern, 1 Matern + nugget */
    int metric;
};

#define XG_GC_ROWS 8
/* one CTA: XG_GC_ROWS rows of one lower tile of S; partial sums of the four
 * parameters' contractions go to part[4 * blockIdx.x + p] */
__global__ void __launch_bounds__(256) xg_grad_contract_kernel(const double *__restrict__ S,
                                                               const int2 *__restrict__ tile_ij, int nt, int ts,
                                                               const double *__restrict__ x,
                                                               const double *__restrict__ y,
                                                               const double *__restrict__ alpha, int N,
                                                               XgGradParams p, double *__restrict__ part)
{
    __shared__ double red[4][8];
    const int strips = ts / XG_GC_ROWS;
    const long long t = blockIdx.x / strips;
    const int strip = blockIdx.x % strips;
    const int2 ij = tile_ij[t];
    const double *tile = S + t * (long long)ts * ts;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (int rr = 0; rr < XG_GC_ROWS; ++rr) {
        const int r = strip * XG_GC_ROWS + rr;
        const int R = ij.x * ts + r;
        if (R >= N) break;
        const double xr = x[R], yr = y[R], ar = alpha[R];
        for (int c = threadIdx.x; c < ts; c += blockDim.x) {
            const int Cc = ij.y * ts + c;
            if (Cc >= N || Cc > R) continue;
            const double w = (Cc == R ? 0.5 : 1.0) * (ar * alpha[Cc] - tile[(long long)r * ts + c]);
            const double d = xg_distance(xr, yr, x[Cc], y[Cc], p.metric);
            const double rd = d / p.beta;
            if (rd == 0.0) {
                acc[0] += w;                     /* dSigma/dsigma2 = 1 on the zero-distance branch */
                if (p.kernel == 1) acc[3] += w;  /* dSigma/dtau2 */
            } else {
                double m, ds, db, dn;
                xg_matern_grad(rd, p.nu, p.con, p.sigma2, p.beta, p.dlogcon, &m, &ds, &db, &dn);
                acc[0] += w * ds;
                acc[1] += w * db;
                acc[2] += w * dn;
            }
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        double v = acc[q];
        for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        if (lane == 0) red[q][warp] = v;
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        double v = 0.0;
        for (int w = 0; w < 8; ++w) v += red[threadIdx.x][w];
        part[4 * (long long)blockIdx.x + threadIdx.x] = v;
    }
}

/* deterministic final sum of the per-CTA partials */
__global__ void xg_grad_reduce_kernel(const double *part, long long nblocks, double *out)
{
    __shared__ double red[4][32];
    const int p = threadIdx.y; /* 4 x 32 threads */
    double v = 0.0;
    for (long long b = threadIdx.x; b < nblocks; b += 32) v += part[4 * b + p];
    red[p][threadIdx.x] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int i = 0; i < 32; ++i) s += red[p][i];
        out[p] = s;
    }
}

/* ========================================================================== */
/* launchers                                                                  */
/* ========================================================================== */

size_t xg_tile_gemm_smem_bytes() { return (size_t)XG_TG_STAGES * XG_TG_STAGE_BYTES + 2 * XG_TG_STAGES * 8 + 1024; }

cudaError_t xg_gradient_kernels_configure()
{
    return cudaFuncSetAttribute(xg_tile_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)xg_tile_gemm_smem_bytes());
}

void xg_launch_zero_diag(double *X, int nt, int ts, cudaStream_t st)
{
    xg_zero_diag_kernel<<<dim3(16, nt), 256, 0, st>>>(X, nt, ts);
}

long long xg_grad_contract_blocks(long long ntiles, int ts) { return ntiles * (ts / XG_GC_ROWS); }

void xg_launch_grad_contract(const double *S, const int2 *tile_ij, long long ntiles, int nt, int ts, const double *x,
                             const double *y, const double *alpha, int N, const XgMaternParams &mp, int kernel,
                             int metric, double dlogcon, double *tab, double *part, double *out, cudaStream_t st)
{
    if (tab && xg_tab_covers(mp, N)) {
        xg_launch_grad_tables(mp, dlogcon, tab, st);
        xg_launch_grad_contract_tab(S, ntiles, nt, ts, x, y, alpha, N, mp, kernel, metric, dlogcon, tab, part, st);
        xg_grad_reduce_kernel<<<1, dim3(32, 4), 0, st>>>(part, xg_grad_contract_tab_blocks(ntiles, ts), out);
        return;
    }
    XgGradParams p;
    p.sigma2 = mp.sigma2;
    p.beta = mp.beta;
    p.nu = mp.nu;
    p.nugget = mp.nugget;
    p.con = mp.con;
    p.dlogcon = dlogcon;
    p.kernel = kernel;
    p.metric = metric;
    const long long blocks = xg_grad_contract_blocks(ntiles, ts);
    xg_grad_contract_kernel<<<(unsigned)blocks, 256, 0, st>>>(S, tile_ij, nt, ts, x, y, alpha, N, p, part);
    xg_grad_reduce_kernel<<<1, dim3(32, 4), 0, st>>>(part, blocks, out);
}

/* C(R, I) = sum_{K >= I} A(R, K) B_slot(K, I)^T: A and C R-layout (C != A),
 * B lower-tile packed.  With B = X (X_IK at slot (K, I)) this is C = A X^T;
 * with B holding the transposed tiles of a factor L, C = A L. */
void xg_launch_rhs_tri_product(const CUtensorMap &mapA, const CUtensorMap &mapB, double *C, int mt, int nt, int ts,
                               int *status, cudaStream_t st)
{
    const int bpt = ts / XG_TG_BM;
    const long long jobs = (long long)mt * nt;
    xg_tile_gemm_kernel<<<(unsigned)(jobs * bpt * bpt), XG_TG_THREADS, xg_tile_gemm_smem_bytes(), st>>>(
        mapA, mapB, C, nt, ts, mt, status);
}
