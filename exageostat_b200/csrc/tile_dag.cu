/*
 * Tile Cholesky in one persistent launch: a dataflow of 128 x 128 blocks.
 *
 * The per-step launches (POTRF, panel TRSM, trailing update per tile column)
 * leave a small or mid-size factorisation waiting on launch gaps, on kernels
 * of a few CTAs, and on reading and writing every trailing block once per
 * step.  Here block (I, J) of the factor is ONE task of one CTA:
 *
 *   C = A_IJ - sum_{K < J} L_IK L_JK^T     TMA-fed DMMA, C in registers throughout
 *                                          (K >= J0 in a window of columns J0 .. : the
 *                                          panels of the INT8 path, whose earlier columns
 *                                          are already applied)
 *   I == J: L_JJ = chol(C) (xg_potrf128), log-det, forward solve of v_J
 *   I >  J: L_IJ = C L_JJ^-T in the same registers, v_I -= L_IJ v_J
 *
 * so each block is read and written once (left-looking).  Tasks are taken in
 * block-column order from one counter; a task waits, block by block, for the
 * flags of the operands it is about to read, so a CTA runs ahead into later
 * columns as far as its operands are ready, and the serial chain per column
 * is POTRF -> TRSM of one block -> the last product of the next diagonal
 * block.  A task waits only on tasks taken earlier by a running CTA: the
 * launch cannot deadlock.  Every wait is bounded.
 *
 * The blocks are sub-blocks of the stored ts x ts tiles (ts a multiple of
 * 128), so the layout of the factor is the one every other kernel reads;
 * blocks that are padding only (rows past N) already hold the identity and
 * are no tasks.  Replaces CHAMELEON_dpotrf_Tile with core_dmdet and the Z
 * solve of MLE_dexact.c:372-391 (the StarPU task graph of psdportf.c:85-186
 * with an infinite band).
 */
#include <math.h>
#include <stdint.h>

#include "xg_common.cuh"
#include "xg_dag.cuh"
#include "xg_kernels.h"
#include "xg_potrf128.cuh"

#define XG_D_STAGES 4
#define XG_D_RING_BYTES (XG_D_STAGES * XG_D_STAGE_BYTES)
/* the triangle and the inverses (xg_dag.cuh), v_J */
#define XG_D_TRSM_BYTES (XG_D_TRI_BYTES + XG_SUB * 8)
#define XG_D_POTRF_BYTES (XG_P_DOUBLES * 8)
#define XG_D_MAX2(a, b) ((a) > (b) ? (a) : (b))
#define XG_D_AREA_BYTES XG_D_MAX2(XG_D_RING_BYTES, XG_D_MAX2(XG_D_TRSM_BYTES, XG_D_POTRF_BYTES))
#define XG_D_SMEM (1024 + XG_D_AREA_BYTES + 128)

__global__ void __launch_bounds__(XG_D_THREADS, 1)
    xg_tile_dag_kernel(const __grid_constant__ CUtensorMap map, XgDag G)
{
    extern __shared__ __align__(1024) unsigned char xg_smem_raw[];
    unsigned char *smem = (unsigned char *)(((uintptr_t)xg_smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t *full = (uint64_t *)(smem + XG_D_AREA_BYTES);
    uint64_t *empty = full + XG_D_STAGES;
    uint64_t *lbar = empty + XG_D_STAGES; /* the triangle and inverses of L_JJ have landed */
    __shared__ long long s_task;
    __shared__ int s_skip, s_bad;
    __shared__ double s_sums[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, tq = lane & 3;
    /* 16-row strip of the block owned by this warp: paired so that the two
     * warps of a scheduler share a diagonal block's triangle evenly */
    const int strip = warp < 4 ? warp : 11 - warp;
    const int r0 = strip * 16 + g;
    const int ts = G.ts, b = ts / XG_SUB;
    if (tid == 0) {
        for (int s = 0; s < XG_D_STAGES; ++s) {
            xg_mbar_init(&full[s], 1);
            xg_mbar_init(&empty[s], XG_D_THREADS / 32);
        }
        xg_mbar_init(lbar, 1);
        xg_fence_barrier_init();
        xg_prefetch_tensormap(&map);
        s_bad = 0;
    }
    uint32_t it0 = 0, lphase = 0; /* slabs of all tasks so far; phase of lbar */
    for (;;) {
        __syncthreads(); /* the previous task is finished by every thread */
        if (tid == 0) {
            long long q = -1;
            if (!*(volatile int *)G.abort) {
                q = (long long)atomicAdd(G.next, 1u);
                if (q >= G.ntasks) q = -1;
            }
            s_task = q;
        }
        __syncthreads();
        const long long q = s_task;
        if (q < 0) break;
        int f = 0, I, J;
        if (G.tasks) {
            const int4 t = G.tasks[q];
            f = t.x;
            I = t.y;
            J = t.z;
        } else {
            const int2 t = xg_tile_decode_fast(q + xg_tile_index(G.J0, G.J0, G.one.nb), G.one.nb);
            I = t.x;
            J = t.y;
        }
        const XgDagField fd = G.tasks ? G.F[f] : G.one;
        const int nt = fd.nt, nb = fd.nb;
        const bool diag = I == J;
        int *status = G.status + 2 * f;
        int *flags = G.flags + fd.flag_off;
        const int *flagI = flags, *flagJ = flags;
        const int i = I / b, j = J / b;
        double *C = G.data + (fd.tile_off + xg_tile_index(i, j, nt)) * (long long)ts * ts +
                    (long long)(I % b * XG_SUB) * ts + J % b * XG_SUB;
        double *dinv = G.dinv + fd.dinv_off * 32 + (long long)J * XG_SUB * 32;
        double *v = G.v ? G.v + fd.vec_off : nullptr;
        if (tid == 0) s_skip = *(volatile int *)status != 0;
        __syncthreads();
        if (!s_skip) {
            /* ---- C = A_IJ - sum_K L_IK L_JK^T: accumulators hold -C ---- */
            const int nlim = diag ? 2 * strip + 2 : 16; /* 8-column groups: a diagonal block's lower part */
            double acc[16][4];
#pragma unroll
            for (int n = 0; n < 16; ++n)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    double2 c = make_double2(0.0, 0.0);
                    if (n < nlim)
                        c = __ldcg(reinterpret_cast<const double2 *>(C + (long long)(r0 + 8 * h) * ts + 8 * n + 2 * tq));
                    acc[n][2 * h] = -c.x;
                    acc[n][2 * h + 1] = -c.y;
                }
            const int KT = (J - G.J0) * (XG_SUB / XG_D_BK);
            int issued = 0, ready = G.J0; /* thread 0: slabs issued; operand blocks known to be finished */
            bool ok = true;
            /* the slabs reuse shared memory that generic accesses touched */
            xg_fence_proxy_async();
            __syncthreads();
            for (int kb = 0; kb < KT; ++kb) {
                if (tid == 0) {
                    while (issued < KT && issued < kb + XG_D_STAGES) {
                        const int kblk = G.J0 + issued / (XG_SUB / XG_D_BK);
                        if (kblk >= ready) {
                            const int *pi = flagI + xg_tile_index(I, kblk, nb), *pj = flagJ + xg_tile_index(J, kblk, nb);
                            /* with slabs in flight an unfinished operand is looked at again after
                             * the next one; with none it is waited for */
                            if (issued > kb) {
                                if (!xg_dag_acquire(pi) || !xg_dag_acquire(pj)) break;
                            } else if (!xg_dag_wait(pi, G.abort) || !xg_dag_wait(pj, G.abort)) {
                                ok = false;
                                break;
                            }
                            ready = kblk + 1;
                            asm volatile("fence.proxy.async.global;" ::: "memory");
                        }
                        const uint32_t s = (it0 + issued) % XG_D_STAGES, use = (it0 + issued) / XG_D_STAGES;
                        if (use > 0 && !xg_mbar_wait(&empty[s], (use - 1) & 1)) {
                            ok = false;
                            break;
                        }
                        const int k = kblk / b, kx = kblk % b * XG_SUB + issued % (XG_SUB / XG_D_BK) * XG_D_BK;
                        unsigned char *sa = smem + s * XG_D_STAGE_BYTES;
                        xg_mbar_arrive_expect_tx(&full[s], diag ? XG_D_BOX_BYTES : XG_D_STAGE_BYTES);
                        xg_tma_load_2d(sa, &map, kx,
                                       (int)((fd.tile_off + xg_tile_index(i, k, nt)) * ts + I % b * XG_SUB), &full[s]);
                        if (!diag)
                            xg_tma_load_2d(sa + XG_D_BOX_BYTES, &map, kx,
                                           (int)((fd.tile_off + xg_tile_index(j, k, nt)) * ts + J % b * XG_SUB),
                                           &full[s]);
                        ++issued;
                    }
                    if (!ok) *(volatile int *)&s_bad = 1;
                }
                __syncwarp();
                if (*(volatile int *)&s_bad) ok = false;
                const uint32_t s = (it0 + kb) % XG_D_STAGES;
                if (ok && !xg_mbar_wait(&full[s], ((it0 + kb) / XG_D_STAGES) & 1)) ok = false;
                if (!__all_sync(0xffffffffu, ok)) {
                    ok = false;
                    *(volatile int *)&s_bad = 1;
                    break;
                }
                const unsigned char *sa = smem + s * XG_D_STAGE_BYTES;
                const unsigned char *sb = diag ? sa : sa + XG_D_BOX_BYTES;
                xg_dag_slab(acc, sa, sb, r0, g, tq, nlim);
                __syncwarp();
                if (lane == 0) xg_mbar_arrive(&empty[s]);
            }
            __syncthreads();
            if (s_bad) {
                /* copies in flight land before the CTA may exit */
                if (tid == 0) {
                    atomicOr(status, XG_ST_TIMEOUT);
                    atomicExch(G.abort, 1);
                    for (int u = issued > XG_D_STAGES ? issued - XG_D_STAGES : 0; u < issued; ++u)
                        xg_mbar_wait(&full[(it0 + u) % XG_D_STAGES], ((it0 + u) / XG_D_STAGES) & 1);
                }
                return;
            }
            it0 += KT;
            if (diag) {
                /* ---- L_JJ, v_J, log-det ---- */
                double *S = (double *)smem;
                double *W = S + XG_SUB * XG_P_LDS, *X = W + (XG_SUB / XG_P_NB) * XG_P_WSZ, *vs = X + 2 * XG_P_WSZ;
#pragma unroll
                for (int n = 0; n < 16; ++n)
                    if (n < nlim)
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            *reinterpret_cast<double2 *>(S + (r0 + 8 * h) * XG_P_LDS + 8 * n + 2 * tq) =
                                make_double2(-acc[n][2 * h], -acc[n][2 * h + 1]);
                if (v && tid < XG_SUB) vs[tid] = __ldcg(v + J * XG_SUB + tid);
                /* zeros to the right of L_JJ in its tile */
                const int right = (ts - (J % b + 1) * XG_SUB) / 2;
                for (int r = warp; r < XG_SUB; r += XG_D_THREADS / 32)
                    for (int c = lane; c < right; c += 32)
                        *reinterpret_cast<double2 *>(C + (long long)r * ts + XG_SUB + 2 * c) = make_double2(0.0, 0.0);
                const int fail = xg_potrf128(S, W, X, vs, v != nullptr, C, ts, dinv, s_sums);
                if (fail) {
                    if (tid == 0) {
                        atomicCAS(status + 1, 0, J * XG_SUB + fail);
                        atomicOr(status, XG_ST_NOT_SPD);
                    }
                } else {
                    if (v && tid < XG_SUB) v[J * XG_SUB + tid] = vs[tid];
                    if (tid == 0) {
                        G.part[fd.part_off + J] = s_sums[0];
                        if (v) G.part[fd.part_off + nb + J] = s_sums[1];
                    }
                }
            } else {
                /* ---- L_IJ = C L_JJ^-T: L_JJ (as operand boxes) and the inverses of its
                 * 32 x 32 diagonal blocks into shared memory, then each warp solves its
                 * 16 rows in registers ---- */
                const double *DS = (const double *)(smem + XG_D_TRI_BOXES * XG_D_BOX_BYTES);
                double *VS = (double *)(smem + XG_D_TRI_BYTES); /* [128] v_J */
                if (tid == 0) {
                    if (xg_dag_wait(flagJ + xg_tile_index(J, J, nb), G.abort)) {
                        const int row = (int)((fd.tile_off + xg_tile_index(j, j, nt)) * ts + J % b * XG_SUB);
                        asm volatile("fence.proxy.async;" ::: "memory");
                        xg_mbar_arrive_expect_tx(lbar, XG_D_TRI_BYTES + (v ? XG_SUB : 0) * 8);
                        xg_dag_load_tri(smem, &map, J % b * XG_SUB, row, dinv, lbar);
                        if (v) xg_bulk_load(VS, v + J * XG_SUB, XG_SUB * 8, lbar);
                    } else {
                        *(volatile int *)&s_bad = 1;
                    }
                }
                __syncthreads();
                if (!s_bad && !xg_mbar_wait(lbar, lphase)) *(volatile int *)&s_bad = 2;
                lphase ^= 1;
                __syncthreads();
                if (s_bad) {
                    if (tid == 0) {
                        atomicOr(status, XG_ST_TIMEOUT);
                        atomicExch(G.abort, 1);
                        if (s_bad == 2) xg_mbar_wait(lbar, lphase ^ 1);
                    }
                    return;
                }
                xg_dag_solve(acc, smem, DS, C, ts, r0, g, tq);
                if (v) {
                    double t0 = 0.0, t1 = 0.0;
#pragma unroll
                    for (int n = 0; n < 16; ++n) {
                        const double2 w = *reinterpret_cast<const double2 *>(VS + 8 * n + 2 * tq);
                        t0 = fma(acc[n][0], w.x, fma(acc[n][1], w.y, t0));
                        t1 = fma(acc[n][2], w.x, fma(acc[n][3], w.y, t1));
                    }
                    for (int o = 1; o < 4; o <<= 1) {
                        t0 += __shfl_xor_sync(0xffffffffu, t0, o);
                        t1 += __shfl_xor_sync(0xffffffffu, t1, o);
                    }
                    if (tq == 0) {
                        double *vi = v + I * XG_SUB + r0;
                        vi[0] = __ldcg(vi) - t0;
                        vi[8] = __ldcg(vi + 8) - t1;
                    }
                }
            }
        }
        /* publish: every thread's stores, then the flag (also for a field that
         * has failed: its later tasks skip their bodies) */
        asm volatile("fence.proxy.async.global;" ::: "memory");
        __threadfence();
        __syncthreads();
        if (tid == 0) xg_dag_release(flags + xg_tile_index(I, J, nb));
    }
}

cudaError_t xg_dag_kernels_configure()
{
    return cudaFuncSetAttribute(xg_tile_dag_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, XG_D_SMEM);
}

void xg_launch_dag(const CUtensorMap &map, const XgDag &G, int max_ctas, cudaStream_t st)
{
    if (G.ntasks <= 0) return;
    const unsigned grid = (unsigned)(G.ntasks < max_ctas ? G.ntasks : max_ctas);
    xg_tile_dag_kernel<<<grid, XG_D_THREADS, XG_D_SMEM, st>>>(map, G);
}
