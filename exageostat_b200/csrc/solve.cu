/*
 * Memory-bound kernels on the lower-tile factor and the kriging kernels.
 *
 *   xg_trmv_lower_kernel      z = L e (CHAMELEON_dtrmm_Tile(Left, Lower, NoTrans, NonUnit),
 *                             exageostat_exact/src/compute/MLE_dexact.c:120)
 *   xg_trsv_lt_*              alpha = L^-T v, the backward half of CHAMELEON_dposv_Tile (MLE_dexact.c:812)
 *   xg_predict_cross_kernel   zmiss = Sigma(miss, obs) alpha with the cross-covariance generated on the
 *                             fly (dcmg of C12 + CHAMELEON_dgemm_Tile, MLE_dexact.c:803-820), never stored
 *   xg_mse_kernel             sum (zactual - zmiss)^2 / nmiss (CORE_dmse_starpu,
 *                             runtime/starpu/codelets/codelet_zmse.c:22-38; MLE_dexact.c:845)
 */
#include <math.h>

#include "kbessel.cuh"
#include "xg_common.cuh"
#include "xg_kernels.h"
#include "xg_matern.cuh"

/* ---- z = L e : 32 rows of tile-row i per CTA, 8 warps x 4 rows ---- */
__global__ void __launch_bounds__(256) xg_trmv_lower_kernel(XgTileArgs T, const double *__restrict__ e,
                                                            double *__restrict__ z, const int *status)
{
    if (*status != 0) return;
    const int ts = T.ts;
    const int strips = ts / 32;
    const int i = blockIdx.x / strips, strip = blockIdx.x % strips;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (int j = 0; j <= i; ++j) {
        const double *tile = T.data + xg_tile_index(i, j, T.nt) * (long long)ts * ts;
        const double *ej = e + (long long)j * ts;
        for (int c = lane; c < ts; c += 32) {
            const double ec = ej[c];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = strip * 32 + warp * 4 + q;
                acc[q] += tile[(long long)r * ts + c] * ec;
            }
        }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        double s = acc[q];
        for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        if (lane == 0) z[(long long)i * ts + strip * 32 + warp * 4 + q] = s;
    }
}

void xg_launch_trmv_lower(const XgTileArgs &T, const double *e, double *z, const int *status, cudaStream_t st)
{
    xg_trmv_lower_kernel<<<T.nt * (T.ts / 32), 256, 0, st>>>(T, e, z, status);
}

/* ---- alpha = L^-T v ---- */

#define XG_TL_THREADS 256
#define XG_TL_LDS 130 /* row stride of the staged L_JJ */
#define XG_TL_SMEM ((128 * XG_TL_LDS + 128 * 33 + 8 * 128 + 128 + 128) * 8)

__device__ __forceinline__ bool xg_trsv_wait(const int *p, const int *abort)
{
    int v;
    const uint64_t t0 = xg_globaltimer_ns();
    for (uint32_t it = 1;; ++it) {
        asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
        if (v) return true;
        if ((it & 63u) == 0u &&
            (*(volatile const int *)abort || xg_globaltimer_ns() - t0 > 2000000000ull))
            return false;
    }
}

/* Block column J of the backward solve is one task of one CTA:
 *   w = v_J - sum_{I > J} L_IJ^T a_I  (I from the last block up), a_J = L_JJ^-T w.
 * Persistent CTAs take the columns from the last one down, so a task waits
 * only on tasks taken earlier.  The entries of a block are in registers
 * before its a_I is waited for, and L_JJ with the inverses of its 32 x 32
 * diagonal blocks in shared memory before the first wait, so the serial chain
 * per 128 rows is one flag, one 128-term product and four 32-row steps.
 * Bound: the chain (about 5 us per 128 rows), and one read of L for large N;
 * the launches per tile row that this replaces took 230 us (ts = 256) to
 * 450 us (ts = 512) each for the serial substitution in the diagonal tile. */
__global__ void __launch_bounds__(XG_TL_THREADS, 1) xg_trsv_lt_kernel(XgTrsv G)
{
    extern __shared__ __align__(16) double xg_smem_d[];
    double *LS = xg_smem_d;             /* [128][130] L_JJ */
    double *DS = LS + 128 * XG_TL_LDS;  /* [128][33] its inverted 32 x 32 diagonal blocks */
    double *red = DS + 128 * 33;        /* [8][128] */
    double *w = red + 8 * 128;          /* [128] */
    double *a = w + 128;                /* [128] */
    __shared__ long long s_task;
    __shared__ int s_skip, s_bad;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ts = G.ts, b = ts / 128;
    if (tid == 0) s_bad = 0;
    for (;;) {
        __syncthreads();
        if (tid == 0) {
            long long q = (long long)atomicAdd(G.next, 1u);
            if (q >= G.ntasks || *(volatile int *)G.abort) q = -1;
            s_task = q;
        }
        __syncthreads();
        const long long q = s_task;
        if (q < 0) break;
        const int2 t = G.tasks ? G.tasks[q] : make_int2(0, G.one.nb - 1 - (int)q);
        const int f = t.x, J = t.y;
        const XgDagField fd = G.tasks ? G.F[f] : G.one;
        const int nt = fd.nt, nb = fd.nb, j = J / b, cj = J % b * 128;
        int *flags = G.flags + fd.tflag_off;
        double *v = G.v + fd.vec_off;
        if (tid == 0) s_skip = *(volatile int *)(G.status + 2 * f) != 0;
        __syncthreads();
        if (s_skip) continue; /* the whole field is skipped: nobody waits for the flag */
        const double *Ljj = G.data + (fd.tile_off + xg_tile_index(j, j, nt)) * (long long)ts * ts + (long long)cj * ts + cj;
        const double *D = G.dinv + (fd.dinv_off + (long long)J * 128) * 32;
#pragma unroll 8
        for (int u = 0; u < 32; ++u) {
            const int idx = tid + u * XG_TL_THREADS, r = idx >> 6, c = idx & 63;
            const double2 x = *(reinterpret_cast<const double2 *>(Ljj + (long long)r * ts) + c);
            *reinterpret_cast<double2 *>(LS + r * XG_TL_LDS + 2 * c) = x;
        }
#pragma unroll 8
        for (int u = 0; u < 16; ++u) {
            const int idx = tid + u * XG_TL_THREADS;
            DS[(idx >> 5) * 33 + (idx & 31)] = D[idx];
        }
        if (tid < 128) w[tid] = v[J * 128 + tid];
        /* warp: rows 16 warp .. + 15 of each block; lane: columns 2 lane, + 1, 64 + 2 lane, + 1 */
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        bool ok = true;
        for (int I = nb - 1; I > J && ok; --I) {
            const int i = I / b;
            const double *T = G.data + (fd.tile_off + xg_tile_index(i, j, nt)) * (long long)ts * ts +
                              (long long)(I % b * 128 + 16 * warp) * ts + cj + 2 * lane;
            double2 x[16][2];
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                x[r][0] = *reinterpret_cast<const double2 *>(T + (long long)r * ts);
                x[r][1] = *reinterpret_cast<const double2 *>(T + (long long)r * ts + 64);
            }
            if (lane == 0) ok = xg_trsv_wait(flags + I, G.abort);
            ok = __shfl_sync(0xffffffffu, ok, 0);
            __syncwarp(); /* lane 0's acquire orders the other lanes' loads */
            double av = 0.0;
            if (lane < 16)
                asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];"
                             : "=d"(av)
                             : "l"(v + I * 128 + 16 * warp + lane)
                             : "memory");
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                const double ar = __shfl_sync(0xffffffffu, av, r);
                acc[0] = fma(x[r][0].x, ar, acc[0]);
                acc[1] = fma(x[r][0].y, ar, acc[1]);
                acc[2] = fma(x[r][1].x, ar, acc[2]);
                acc[3] = fma(x[r][1].y, ar, acc[3]);
            }
        }
        if (!ok) s_bad = 1;
        *reinterpret_cast<double2 *>(red + warp * 128 + 2 * lane) = make_double2(acc[0], acc[1]);
        *reinterpret_cast<double2 *>(red + warp * 128 + 64 + 2 * lane) = make_double2(acc[2], acc[3]);
        __syncthreads();
        if (s_bad) {
            if (tid == 0) {
                atomicOr(G.status + 2 * f, XG_ST_TIMEOUT);
                atomicExch(G.abort, 1);
            }
            return;
        }
        if (tid < 128) {
            double sum = 0.0;
#pragma unroll
            for (int u = 0; u < 8; ++u) sum += red[u * 128 + tid];
            w[tid] -= sum;
        }
        __syncthreads();
        /* a_JJ block by block from the bottom: a_q = D_q^T w_q, then w above -= L_q^T a_q */
#pragma unroll 1
        for (int qb = 3; qb >= 0; --qb) {
            if (warp == 0) {
                double s0 = 0.0, s1 = 0.0;
#pragma unroll
                for (int r = 0; r < 32; r += 2) {
                    s0 = fma(DS[(32 * qb + r) * 33 + lane], w[32 * qb + r], s0);
                    s1 = fma(DS[(32 * qb + r + 1) * 33 + lane], w[32 * qb + r + 1], s1);
                }
                a[32 * qb + lane] = s0 + s1;
            }
            __syncthreads();
            if (warp < qb) {
                double s0 = w[32 * warp + lane], s1 = 0.0;
#pragma unroll
                for (int r = 0; r < 32; r += 2) {
                    s0 = fma(-LS[(32 * qb + r) * XG_TL_LDS + 32 * warp + lane], a[32 * qb + r], s0);
                    s1 = fma(-LS[(32 * qb + r + 1) * XG_TL_LDS + 32 * warp + lane], a[32 * qb + r + 1], s1);
                }
                w[32 * warp + lane] = s0 + s1;
            }
            __syncthreads();
        }
        if (tid < 128) {
            v[J * 128 + tid] = a[tid];
            __threadfence();
        }
        __syncthreads();
        if (tid == 0) asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(flags + J), "r"(1) : "memory");
    }
}

cudaError_t xg_solve_kernels_configure()
{
    return cudaFuncSetAttribute(xg_trsv_lt_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, XG_TL_SMEM);
}

void xg_launch_trsv_lower_t(const XgTrsv &G, int max_ctas, cudaStream_t st)
{
    if (G.ntasks <= 0) return;
    const unsigned grid = (unsigned)(G.ntasks < max_ctas ? G.ntasks : max_ctas);
    xg_trsv_lt_kernel<<<grid, XG_TL_THREADS, XG_TL_SMEM, st>>>(G);
}

/* ---- kriging: zmiss[m] = sum_o Sigma(miss_m, obs_o) alpha_o ---- */
__global__ void __launch_bounds__(256) xg_predict_cross_kernel(const double *__restrict__ xm,
                                                               const double *__restrict__ ym, int nmiss,
                                                               const double *__restrict__ xo,
                                                               const double *__restrict__ yo, int nobs,
                                                               const double *__restrict__ alpha, XgMaternParams p,
                                                               int metric, double *__restrict__ zmiss)
{
    __shared__ double red[8];
    const int m = blockIdx.x;
    double s = 0.0;
    if (p.bivariate) {
        /* rows and columns interleave the two variables: index 2 l + v */
        const double x1 = xm[m >> 1], y1 = ym[m >> 1];
        for (int o = threadIdx.x; o < nobs; o += blockDim.x)
            s += xg_matern_value_biv(xg_distance(x1, y1, xo[o >> 1], yo[o >> 1], metric), p, m & 1, o & 1) * alpha[o];
    } else {
        const double x1 = xm[m], y1 = ym[m];
        for (int o = threadIdx.x; o < nobs; o += blockDim.x)
            s += xg_matern_value(xg_distance(x1, y1, xo[o], yo[o], metric), p) * alpha[o];
    }
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < 8; ++w) t += red[w];
        zmiss[m] = t;
    }
}

void xg_launch_predict_cross(const double *xm, const double *ym, int nmiss, const double *xo, const double *yo,
                             int nobs, const double *alpha, const XgMaternParams &p, int metric, double *zmiss,
                             cudaStream_t st)
{
    if (nmiss <= 0) return;
    xg_predict_cross_kernel<<<nmiss, 256, 0, st>>>(xm, ym, nmiss, xo, yo, nobs, alpha, p, metric, zmiss);
}

__global__ void xg_mse_kernel(const double *__restrict__ za, const double *__restrict__ zm, int n, double *out)
{
    /* out[0] = the MSE; out[1], out[2] = the MSEs of the even and odd entries
     * (the two variables of a bivariate field, CORE_dmse_bivariate_starpu,
     * codelet_zmse_bivariate.c:22-51, averaged over n / 2 as MLE_dexact.c:845-847).
     * blockDim is even, so each thread sees entries of one parity only. */
    __shared__ double red[2][32];
    double s = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double d = za[i] - zm[i];
        s += d * d;
    }
    double se = (threadIdx.x & 1) ? 0.0 : s, so = (threadIdx.x & 1) ? s : 0.0;
    for (int off = 16; off > 0; off >>= 1) {
        se += __shfl_xor_sync(0xffffffffu, se, off);
        so += __shfl_xor_sync(0xffffffffu, so, off);
    }
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = se;
        red[1][threadIdx.x >> 5] = so;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double te = 0.0, to = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            te += red[0][w];
            to += red[1][w];
        }
        out[0] = (te + to) / n;
        const int half = n / 2;
        out[1] = half > 0 ? te / half : 0.0;
        out[2] = half > 0 ? to / half : 0.0;
    }
}

void xg_launch_mse(const double *zactual, const double *zmiss, int nmiss, double *out, cudaStream_t st)
{
    xg_mse_kernel<<<1, 1024, 0, st>>>(zactual, zmiss, nmiss, out);
}

/* ---- element-wise Matern of location pairs (diagnostics and tests) ---- */
__global__ void xg_matern_pairs_kernel(const double *x1, const double *y1, const double *x2, const double *y2, int n,
                                       XgMaternParams p, int metric, double *out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = xg_matern_value(xg_distance(x1[i], y1[i], x2[i], y2[i], metric), p);
}

void xg_launch_matern_pairs(const double *x1, const double *y1, const double *x2, const double *y2, int n,
                            const XgMaternParams &p, int metric, double *out, cudaStream_t st)
{
    if (n <= 0) return;
    xg_matern_pairs_kernel<<<(n + 255) / 256, 256, 0, st>>>(x1, y1, x2, y2, n, p, metric, out);
}

__global__ void xg_bessel_kernel(const double *nu, const double *x, int n, double *out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = xg_bessel_knu(nu[i], x[i]);
}

void xg_launch_bessel(const double *nu, const double *x, int n, double *out, cudaStream_t st)
{
    if (n <= 0) return;
    xg_bessel_kernel<<<(n + 255) / 256, 256, 0, st>>>(nu, x, n, out);
}
