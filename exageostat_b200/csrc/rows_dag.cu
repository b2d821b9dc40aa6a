/*
 * Many right-hand sides against a tile Cholesky factor in one persistent
 * launch, as a dataflow of 128 x 128 blocks (the same blocks and pieces as
 * tile_dag.cu).
 *
 *   XG_ROWS_INVERSE  X L^T = I (X = L^-T, upper triangular, X_IK at packed tile slot (K, I)), then
 *                    S = X X^T written over the factor: the inverse and product of the adjoint
 *                    gradient (steps 2 and 3 of gradient_fp64.cu);
 *                    a window of columns J0 .. : the sums over K < J0 are in place already
 *                    and there are no products (the INT8 path)
 *   XG_ROWS_RHS      Y L^T = B for row blocks in R layout (tile (R, K) at slot K mt + R), up to
 *                    three systems at once: the forward solves of MLOE / MMOM (MLE_dexact.c:1300-1364)
 *                    and the two-sided solves of the Fisher matrix (the second with the lower
 *                    blocks only)
 *
 * Solve task (I, J): Y_IJ = (B_IJ - sum_{K < J} Y_IK L_JK^T) L_JJ^-T with the
 * accumulators in registers from the first product to the store, so a block
 * is written once (the per-step launches it replaces read and wrote every
 * block per step and solved 32-row strips by serial substitution, 105 us a
 * launch at 8 % of the DMMA rate).  A row's blocks wait for the row's earlier
 * ones only; L_JJ is fetched while the products run.  Product task (I, J),
 * J <= I: S_IJ = sum_{K >= I} X_IK X_JK^T, accumulated as the columns of X
 * appear; before the store it waits for every X_RI, R <= J, whose task may
 * still read L_IJ.  Tasks are taken in an order in which each waits only on
 * earlier ones; every wait is bounded.
 */
#include <math.h>
#include <stdint.h>

#include "xg_common.cuh"
#include "xg_dag.cuh"
#include "xg_kernels.h"

/* three stages, so that L_JJ has shared memory of its own beside the ring */
#define XG_R_STAGES 3
#define XG_R_RING_BYTES (XG_R_STAGES * XG_D_STAGE_BYTES)
#define XG_R_SMEM (1024 + XG_R_RING_BYTES + XG_D_TRI_BYTES + 128)

template <int MODE>
__global__ void __launch_bounds__(XG_D_THREADS, 1) xg_rows_dag_kernel(const __grid_constant__ XgRowsMaps M, XgRows G)
{
    extern __shared__ __align__(1024) unsigned char xg_smem_raw[];
    unsigned char *smem = (unsigned char *)(((uintptr_t)xg_smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char *tri = smem + XG_R_RING_BYTES;
    uint64_t *full = (uint64_t *)(tri + XG_D_TRI_BYTES);
    uint64_t *empty = full + XG_R_STAGES;
    uint64_t *lbar = empty + XG_R_STAGES;
    __shared__ long long s_task;
    __shared__ int s_skip, s_bad;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, tq = lane & 3;
    const int r0 = warp * 16 + g;
    const int ts = G.ts, b = ts / XG_DAG_BLOCK;
    constexpr int SPB = XG_DAG_BLOCK / XG_D_BK; /* slabs per block */
    if (tid == 0) {
        for (int s = 0; s < XG_R_STAGES; ++s) {
            xg_mbar_init(&full[s], 1);
            xg_mbar_init(&empty[s], XG_D_THREADS / 32);
        }
        xg_mbar_init(lbar, 1);
        xg_fence_barrier_init();
        s_bad = 0;
    }
    uint32_t it0 = 0, lphase = 0;
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
        long long q = s_task;
        if (q < 0) break;
        int f = 0, sys = 0, I, J;
        bool product = false;
        if (G.tasks) {
            const int4 t = G.tasks[q];
            f = t.x;
            I = t.y;
            J = t.z;
            product = t.w != 0;
        } else if (MODE == XG_ROWS_RHS) {
            sys = (int)(q % G.nsys);
            q /= G.nsys;
            if (G.lower) {
                xg_pair_decode(G.ntasks / G.nsys - 1 - q, &J, &I);
                I = G.one.nb - 1 - I;
                J = G.one.nb - 1 - J;
            } else {
                I = (int)(q % G.one.mr);
                J = (int)(q / G.one.mr);
            }
        } else {
            const long long nx = xg_num_lower_tiles(G.one.nb);
            product = q >= nx;
            if (product)
                xg_pair_decode(q - nx, &I, &J); /* I ascending: the longest sums first */
            else
                xg_pair_decode(q + xg_num_lower_tiles(G.J0), &J, &I);
        }
        const XgRowsField fd = G.tasks ? G.F[f] : G.one;
        const int nt = fd.nt, nb = fd.nb, i = I / b, j = J / b;
        const CUtensorMap *mapY = &M.y[sys], *mapL = &M.l[sys];
        int *flags = G.flags + fd.flag_off + (long long)sys * G.sys_flags;
        int *status = G.status + 2 * f;
        /* flag of block (row I, column K), and the block's place in the tensor */
        auto flag = [&](int row, int K) {
            return flags + (MODE == XG_ROWS_RHS ? (long long)K * fd.mr + row : xg_tile_index(K, row, nb));
        };
        auto slotY = [&](int row, int K) {
            const int ti = row / b, tk = K / b;
            return fd.y_off + (MODE == XG_ROWS_RHS ? (long long)tk * fd.mt + ti : xg_tile_index(tk, ti, nt));
        };
        if (tid == 0) s_skip = *(volatile int *)status != 0;
        __syncthreads();
        if (!s_skip) {
            double *C = product ? G.s + (fd.l_off + xg_tile_index(i, j, nt)) * (long long)ts * ts
                                : G.y[sys] + slotY(I, J) * (long long)ts * ts;
            C += (long long)(I % b * XG_DAG_BLOCK) * ts + J % b * XG_DAG_BLOCK;
            const int k0 = MODE == XG_ROWS_RHS ? 0 : product || I > G.J0 ? I : G.J0, k1 = product ? nb : J;
            const int KT = (k1 - k0) * SPB;
            const bool same = product && I == J; /* both operands are the same rows */
            double acc[16][4];
#pragma unroll
            for (int n = 0; n < 16; ++n)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    double2 c = make_double2(0.0, 0.0);
                    const int r = r0 + 8 * h, cc = 8 * n + 2 * tq;
                    if (MODE == XG_ROWS_RHS || I < G.J0)
                        c = __ldcg(reinterpret_cast<const double2 *>(C + (long long)r * ts + cc));
                    else if (!product && I == J) /* the identity */
                        c = make_double2(r == cc ? 1.0 : 0.0, r == cc + 1 ? 1.0 : 0.0);
                    acc[n][2 * h] = -c.x;
                    acc[n][2 * h + 1] = -c.y;
                }
            /* shared memory last touched by generic reads, next by copies */
            xg_fence_proxy_async();
            __syncthreads();
            int issued = 0, ready = k0;
            bool ok = true;
            if (tid == 0 && !product) {
                xg_mbar_arrive_expect_tx(lbar, XG_D_TRI_BYTES);
                xg_dag_load_tri(tri, mapL, J % b * XG_DAG_BLOCK,
                                (int)((fd.l_off + xg_tile_index(j, j, nt)) * ts + J % b * XG_DAG_BLOCK),
                                G.dinv[sys] + (fd.dinv_off + (long long)J * XG_DAG_BLOCK) * 32, lbar);
            }
            for (int kb = 0; kb < KT; ++kb) {
                if (tid == 0) {
                    while (issued < KT && issued < kb + XG_R_STAGES) {
                        const int K = k0 + issued / SPB;
                        if (K >= ready) {
                            const int *pi = flag(I, K), *pj = product ? flag(J, K) : pi;
                            if (issued > kb) {
                                if (!xg_dag_acquire(pi) || !xg_dag_acquire(pj)) break;
                            } else if (!xg_dag_wait(pi, G.abort) || !xg_dag_wait(pj, G.abort)) {
                                ok = false;
                                break;
                            }
                            ready = K + 1;
                            asm volatile("fence.proxy.async.global;" ::: "memory");
                        }
                        const uint32_t s = (it0 + issued) % XG_R_STAGES, use = (it0 + issued) / XG_R_STAGES;
                        if (use > 0 && !xg_mbar_wait(&empty[s], (use - 1) & 1)) {
                            ok = false;
                            break;
                        }
                        const int kx = K % b * XG_DAG_BLOCK + issued % SPB * XG_D_BK;
                        unsigned char *sa = smem + s * XG_D_STAGE_BYTES;
                        xg_mbar_arrive_expect_tx(&full[s], same ? XG_D_BOX_BYTES : XG_D_STAGE_BYTES);
                        xg_tma_load_2d(sa, mapY, kx, (int)(slotY(I, K) * ts + I % b * XG_DAG_BLOCK), &full[s]);
                        if (!same)
                            xg_tma_load_2d(sa + XG_D_BOX_BYTES, product ? mapY : mapL, kx,
                                           (int)((product ? slotY(J, K) : fd.l_off + xg_tile_index(j, K / b, nt)) * ts +
                                                 J % b * XG_DAG_BLOCK),
                                           &full[s]);
                        ++issued;
                    }
                    if (!ok) *(volatile int *)&s_bad = 1;
                }
                __syncwarp();
                if (*(volatile int *)&s_bad) ok = false;
                const uint32_t s = (it0 + kb) % XG_R_STAGES;
                if (ok && !xg_mbar_wait(&full[s], ((it0 + kb) / XG_R_STAGES) & 1)) ok = false;
                if (!__all_sync(0xffffffffu, ok)) {
                    ok = false;
                    *(volatile int *)&s_bad = 1;
                    break;
                }
                const unsigned char *sa = smem + s * XG_D_STAGE_BYTES;
                xg_dag_slab(acc, sa, same ? sa : sa + XG_D_BOX_BYTES, r0, g, tq, 16);
                __syncwarp();
                if (lane == 0) xg_mbar_arrive(&empty[s]);
            }
            if (product) {
                /* L_IJ may be overwritten once every solve of column I by rows R <= J is done */
                for (int R = tid; R <= J && ok; R += XG_D_THREADS)
                    if (!xg_dag_wait(flag(R, I), G.abort)) {
                        ok = false;
                        *(volatile int *)&s_bad = 1;
                    }
            } else if (ok && !xg_mbar_wait(lbar, lphase)) {
                *(volatile int *)&s_bad = 1;
            }
            __syncthreads();
            if (s_bad) {
                /* copies in flight land before the CTA may exit */
                if (tid == 0) {
                    atomicOr(status, XG_ST_TIMEOUT);
                    atomicExch(G.abort, 1);
                    for (int u = issued > XG_R_STAGES ? issued - XG_R_STAGES : 0; u < issued; ++u)
                        xg_mbar_wait(&full[(it0 + u) % XG_R_STAGES], ((it0 + u) / XG_R_STAGES) & 1);
                    if (!product) xg_mbar_wait(lbar, lphase);
                }
                return;
            }
            it0 += KT;
            if (product) {
#pragma unroll
                for (int n = 0; n < 16; ++n)
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        *reinterpret_cast<double2 *>(C + (long long)(r0 + 8 * h) * ts + 8 * n + 2 * tq) =
                            make_double2(acc[n][2 * h], acc[n][2 * h + 1]);
            } else {
                lphase ^= 1;
                xg_dag_solve(acc, tri, (const double *)(tri + XG_D_TRI_BOXES * XG_D_BOX_BYTES), C, ts, r0, g, tq);
            }
        }
        if (!product) {
            asm volatile("fence.proxy.async.global;" ::: "memory");
            __threadfence();
            __syncthreads();
            if (tid == 0) xg_dag_release(flag(I, J));
        }
    }
}

cudaError_t xg_rows_kernels_configure()
{
    cudaError_t e = cudaFuncSetAttribute(xg_rows_dag_kernel<XG_ROWS_INVERSE>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, XG_R_SMEM);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(xg_rows_dag_kernel<XG_ROWS_RHS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                XG_R_SMEM);
}

void xg_launch_rows(int mode, const XgRowsMaps &M, const XgRows &G, int max_ctas, cudaStream_t st)
{
    if (G.ntasks <= 0) return;
    const unsigned grid = (unsigned)(G.ntasks < max_ctas ? G.ntasks : max_ctas);
    if (mode == XG_ROWS_RHS)
        xg_rows_dag_kernel<XG_ROWS_RHS><<<grid, XG_D_THREADS, XG_R_SMEM, st>>>(M, G);
    else
        xg_rows_dag_kernel<XG_ROWS_INVERSE><<<grid, XG_D_THREADS, XG_R_SMEM, st>>>(M, G);
}
