/*
 * Pieces shared by the block dataflow kernels (tile_dag.cu, rows_dag.cu):
 * flags between CTAs, the 128 x 128 x 16 DMMA step and the triangular solve of
 * a block held in registers.
 *
 * A 128 x 128 block is held by 256 threads as eight 16-row strips, one a
 * warp: acc[n] is the DMMA tile of columns 8 n .. 8 n + 7 (rows g and g + 8
 * of the strip, columns 2 tq and 2 tq + 1), so each warp can solve its rows
 * against L_JJ by itself.  (64 x 32 warp tiles read less shared memory per
 * product, but both are far below its bandwidth.)
 */
#ifndef EXAGEOSTAT_B200_DAG_CUH
#define EXAGEOSTAT_B200_DAG_CUH

#include "xg_common.cuh"
#include "xg_kernels.h"

#define XG_D_BK 16
#define XG_D_THREADS 256
#define XG_D_BOX_BYTES (XG_DAG_BLOCK * XG_D_BK * 8)
#define XG_D_STAGE_BYTES (2 * XG_D_BOX_BYTES)
/* L_JJ as six 128 x 16 boxes (its last 32 columns are not needed), then the
 * inverses of its 32 x 32 diagonal blocks, [128][32] */
#define XG_D_TRI_BOXES 6
#define XG_D_TRI_BYTES (XG_D_TRI_BOXES * XG_D_BOX_BYTES + XG_DAG_BLOCK * 32 * 8)

__device__ __forceinline__ int xg_dag_acquire(const int *p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void xg_dag_release(int *p)
{
    asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(1) : "memory");
}

/* One thread: waits until *p is set; false after 2 s or when another CTA aborted the launch */
__device__ __forceinline__ bool xg_dag_wait(const int *p, const int *abort)
{
    if (xg_dag_acquire(p)) return true;
    const uint64_t t0 = xg_globaltimer_ns();
    for (uint32_t it = 0;; ++it) {
        if (xg_dag_acquire(p)) return true;
        if ((it & 31u) == 31u) {
            if (*(volatile const int *)abort) return false;
            if (xg_globaltimer_ns() - t0 > 2000000000ull) return false;
        }
    }
}

/* acc += A B^T over one 16-wide slab: A the 128 x 16 box at sa (this warp's
 * rows r0 = 16 strip + g and r0 + 8), B the one at sb (rows = columns of acc),
 * both 128-byte swizzled.  k permutation as in xg_gemm_core: lane slot tq
 * holds k = 4 tq .. 4 tq + 3.  nlim: 8-column groups wanted, in fours. */
__device__ __forceinline__ void xg_dag_slab(double (&acc)[16][4], const unsigned char *sa, const unsigned char *sb,
                                            int r0, int g, int tq, int nlim)
{
    /* rows g + 8 m: row & 7 = g */
    const int sw[2] = {((2 * tq) ^ g) << 4, ((2 * tq + 1) ^ g) << 4};
    double2 a0[2], a1[2], bv[2][4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        a0[h] = *(const double2 *)(sa + (r0 << 7) + sw[h]);
        a1[h] = *(const double2 *)(sa + ((r0 + 8) << 7) + sw[h]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) bv[0][u] = *(const double2 *)(sb + ((8 * u + g) << 7) + sw[0]);
#pragma unroll
    for (int n0 = 0; n0 < 16; n0 += 4) {
        /* groups of 32 columns: the branch must skip enough work to stay a
         * branch (skipped by predicates, the DMMAs take their full time) */
        if (n0 >= nlim) break;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            /* the next step's B fragments, in flight under this one's DMMAs */
            const int nn = h ? n0 + 4 : n0;
            if (nn < 16)
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    bv[h ^ 1][u] = *(const double2 *)(sb + ((8 * (nn + u) + g) << 7) + sw[h ^ 1]);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                xg_dmma_16x8x4(acc[n0 + u][0], acc[n0 + u][1], acc[n0 + u][2], acc[n0 + u][3], a0[h].x, a1[h].x,
                               bv[h][u].x);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                xg_dmma_16x8x4(acc[n0 + u][0], acc[n0 + u][1], acc[n0 + u][2], acc[n0 + u][3], a0[h].y, a1[h].y,
                               bv[h][u].y);
        }
    }
}

/* X = T L_JJ^-T for the block with acc = -T, by 32-column blocks: the product
 * with the inverted diagonal block, stored to C (leading dimension ts) and
 * kept in acc, then acc += X L^T for the columns to the right.  The
 * accumulators are the A fragments as they stand: K runs over the columns in
 * the lanes' order, and the B operand is read in the same order.  LS, DS:
 * xg_dag_load_tri. */
__device__ __forceinline__ void xg_dag_solve(double (&acc)[16][4], const unsigned char *LS, const double *DS, double *C,
                                             int ts, int r0, int g, int tq)
{
#pragma unroll
    for (int cb = 0; cb < 4; ++cb) {
        double x[4][4];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
#pragma unroll
            for (int e = 0; e < 4; ++e) x[m][e] = 0.0;
#pragma unroll
            for (int k = 0; k <= m; ++k) { /* D is lower triangular */
                const double2 d = *reinterpret_cast<const double2 *>(DS + (32 * cb + 8 * m + g) * 32 + 8 * k + 2 * tq);
                xg_dmma_16x8x4(x[m][0], x[m][1], x[m][2], x[m][3], acc[4 * cb + k][0], acc[4 * cb + k][2], d.x);
                xg_dmma_16x8x4(x[m][0], x[m][1], x[m][2], x[m][3], acc[4 * cb + k][1], acc[4 * cb + k][3], d.y);
            }
        }
#pragma unroll
        for (int m = 0; m < 4; ++m) {
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[4 * cb + m][e] = -x[m][e];
#pragma unroll
            for (int h = 0; h < 2; ++h)
                *reinterpret_cast<double2 *>(C + (long long)(r0 + 8 * h) * ts + 32 * cb + 8 * m + 2 * tq) =
                    make_double2(acc[4 * cb + m][2 * h], acc[4 * cb + m][2 * h + 1]);
        }
#pragma unroll
        for (int m = 4 * cb + 4; m < 16; ++m)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const double2 l =
                    *reinterpret_cast<const double2 *>(LS + (2 * cb + (k >> 1)) * XG_D_BOX_BYTES +
                                                       ((8 * m + g) << 7) + ((((k & 1) * 4 + tq) ^ g) << 4));
                xg_dmma_16x8x4(acc[m][0], acc[m][1], acc[m][2], acc[m][3], acc[4 * cb + k][0], acc[4 * cb + k][2], l.x);
                xg_dmma_16x8x4(acc[m][0], acc[m][1], acc[m][2], acc[m][3], acc[4 * cb + k][1], acc[4 * cb + k][3], l.y);
            }
    }
}

/* One thread: L_JJ (row and column of its block in the tensor) and its
 * inverses into smem (XG_D_TRI_BYTES); the caller has announced the bytes */
__device__ __forceinline__ void xg_dag_load_tri(unsigned char *smem, const CUtensorMap *map, int x, int row,
                                                const double *dinv, uint64_t *bar)
{
    xg_bulk_load(smem + XG_D_TRI_BOXES * XG_D_BOX_BYTES, dinv, XG_DAG_BLOCK * 32 * 8, bar);
    for (int u = 0; u < XG_D_TRI_BOXES; ++u)
        xg_tma_load_2d(smem + u * XG_D_BOX_BYTES, map, x + u * XG_D_BK, row, bar);
}

#endif
