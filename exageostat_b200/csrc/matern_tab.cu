/*
 * Covariance and derivative tiles of general smoothness from the piecewise
 * polynomial tables of xg_matern_tab.cuh: one small launch builds the tables
 * of an evaluation's parameters, then persistent CTAs keep them in shared
 * memory and fill (or contract) tile strips.
 *
 *   xg_gen_tab_kernel           core_dcmg, core_dcmg_nuggets and the bivariate kernels
 *                               (exageostat_exact/cpu_core/compute/core_zcmg.c:963-994, 1514-1726,
 *                               core_zcmg_nuggets.c:107-156)
 *   xg_grad_contract_tab_kernel the contraction of gradient_fp64.cu's step 4
 *   xg_dsigma_full_tab_kernel   the dSigma/dtheta tiles of the Fisher matrix (MLE_dexact.c:1840-1842)
 *
 * The direct kernels spend 600 to 1300 FP64 operations per element on a series
 * or a quadrature (13-18 G elements/s, ALU bound); a table element costs about
 * 70 and nine shared-memory reads, and its largest error against 30-digit
 * values is 1.5e-15 to 6e-15 over 0.01 <= nu <= 5 (direct: 2e-15 to 2.7e-14,
 * from the rounding of (nu - 1/2) log r - r under the exponential).
 */
#include <math.h>
#include <stdint.h>

#include "xg_common.cuh"
#include "xg_kernels.h"
#include "xg_matern.cuh"
#include "xg_matern_tab.cuh"

/* ========================================================================== */
/* tables                                                                     */
/* ========================================================================== */

/* One warp per three intervals: lane 9 q + j evaluates node j of interval q,
 * then lanes 0 .. 3 nf - 1 form the coefficients of (interval, function). */
template <bool GRAD>
__device__ __forceinline__ void xg_tab_build_warp(double *tab, int i0, double nu, double con, const XgTemme &tm,
                                                  double sigma2, double beta, double dlogcon, double (*f)[3][XG_TAB_NC],
                                                  int lane)
{
    const int q = lane / XG_TAB_NC, j = lane % XG_TAB_NC;
    if (q < 3 && i0 + q < XG_TAB_NINT) {
        double c, hw;
        xg_tab_interval(i0 + q, &c, &hw);
        const double r = xg_tab_node(c, hw, j);
        if (GRAD) {
            double g[3];
            xg_tab_matern_grad(r, nu, con, sigma2, beta, dlogcon, g);
            for (int p = 0; p < 3; ++p) f[p][q][j] = g[p];
        } else {
            f[0][q][j] = xg_tab_matern(r, nu, con, tm);
        }
    }
    __syncwarp();
    const int p = lane / 3, u = lane % 3;
    if (p < (GRAD ? 3 : 1) && i0 + u < XG_TAB_NINT) {
        double c, hw;
        xg_tab_interval(i0 + u, &c, &hw);
        xg_tab_coefficients(f[p][u], hw, tab + (long long)p * XG_TAB_SIZE + (i0 + u) * XG_TAB_NC);
    }
}

struct XgTabFn {
    double nu, con;
    XgTemme tm;
};
struct XgTabFns {
    XgTabFn f[3];
    double sigma2, beta, dlogcon;
};

/* GRAD: the three derivative tables of f[0]; else one Matern table per blockIdx.y */
template <bool GRAD> __global__ void __launch_bounds__(64) xg_tab_build_kernel(double *tab, XgTabFns P)
{
    __shared__ double f[2][3][3][XG_TAB_NC];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i0 = ((int)blockIdx.x * 2 + warp) * 3;
    const XgTabFn &fn = P.f[blockIdx.y];
    xg_tab_build_warp<GRAD>(tab + (long long)blockIdx.y * XG_TAB_SIZE, i0, fn.nu, fn.con, fn.tm, P.sigma2, P.beta,
                            P.dlogcon, f[warp], lane);
}

/* a batch's fields follow the rule of a single field (xg_tab_covers), so their
 * elements are the same */
__device__ __forceinline__ bool xg_tab_wanted(const XgMaternParams &p, int n)
{
    return p.half_integer < 0 && n >= XG_TAB_MIN_N && p.nu <= XG_TAB_NU && xg_tab_scale_ok(p.con) &&
           xg_tab_scale_ok(p.con / p.beta);
}

/* the tables of every field of a batch (blockIdx.y and on by gridDim.y, which
 * the hardware limits to 65535); fields that need none are passed over */
__global__ void __launch_bounds__(64)
    xg_tab_build_batch_kernel(double *tab, const XgBField *__restrict__ F, int nfields)
{
    __shared__ double f[2][3][3][XG_TAB_NC];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int field = (int)blockIdx.y; field < nfields; field += (int)gridDim.y) {
        const XgMaternParams &p = F[field].p;
        if (!xg_tab_wanted(p, F[field].N)) continue;
        __syncwarp(); /* the last field's node values are read */
        xg_tab_build_warp<false>(tab + (long long)field * XG_TAB_SIZE, ((int)blockIdx.x * 2 + warp) * 3, p.nu, p.con,
                                 p.tm, 0.0, 0.0, 0.0, f[warp], lane);
    }
}
#define XG_TAB_BUILD_BLOCKS ((XG_TAB_NINT + 5) / 6)

/* ========================================================================== */
/* generation                                                                 */
/* ========================================================================== */

#define XG_GT_ROWS 8
#define XG_GT_THREADS 256

/* outside the table's range: out of line, a few elements at most */
__device__ __noinline__ double xg_gen_tab_rare(double r, double nu, double con)
{
    return xg_matern_general(r, nu, con);
}

__device__ __forceinline__ double xg_tab_eval(const double *tab, double r, double nu, double con)
{
    const unsigned i = xg_tab_index(r);
    if (i >= XG_TAB_NINT) return xg_gen_tab_rare(r, nu, con);
    return xg_tab_poly(tab, i, r - xg_tab_centre(r)) * exp(-r);
}

__device__ __forceinline__ void xg_tab_stage(double *dst, const double *src, int n)
{
    for (int i = (int)threadIdx.x; i < n / 2; i += (int)blockDim.x)
        reinterpret_cast<double2 *>(dst)[i] = reinterpret_cast<const double2 *>(src)[i];
}

/* one strip of XG_GT_ROWS rows of tile (i, j): each thread two adjacent
 * columns at a time (16-byte stores).  BIV: those are the two variables of
 * one location (matrix index 2 l + v), which share the distance and, with
 * equal scales, the exponential's argument. */
template <bool BIV>
__device__ __forceinline__ void xg_gen_tab_strip(double *tile, int ts, int2 ij, int strip, const double *__restrict__ xr,
                                                 const double *__restrict__ yr, const double *__restrict__ xc,
                                                 const double *__restrict__ yc, int n_rows, int n_cols,
                                                 const XgMaternParams &p, int metric, int identity_pad,
                                                 const double *tab)
{
    const int half = ts / 2;
    for (int e = (int)threadIdx.x; e < XG_GT_ROWS * half; e += XG_GT_THREADS) {
        const int rr = e / half, c = 2 * (e - rr * half), r = strip * XG_GT_ROWS + rr;
        const int R = ij.x * ts + r, C = ij.y * ts + c;
        double v[2];
        if (BIV && R < n_rows && C < n_cols) { /* both variables: n_cols is even */
            const double d = xg_distance(xr[R >> 1], yr[R >> 1], xc[C >> 1], yc[C >> 1], metric);
            const double r0 = d / p.beta;
            const int a = R & 1;
            if (r0 == 0.0) {
                v[0] = a ? p.cross0 : p.sigma2;
                v[1] = a ? p.sigma2b : p.cross0;
            } else {
                const double r12 = p.beta12 == p.beta ? r0 : d / p.beta12;
                const double ra = !a ? r0 : p.beta2 == p.beta ? r0 : d / p.beta2;
                const double same = xg_tab_eval(tab + (a ? XG_TAB_SIZE : 0), ra, a ? p.nu2 : p.nu, a ? p.con2 : p.con);
                const double cross = xg_tab_eval(tab + 2 * XG_TAB_SIZE, r12, p.nu12, p.con12);
                v[0] = a ? cross : same;
                v[1] = a ? same : cross;
            }
        } else {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                if (!BIV && R < n_rows && C + u < n_cols) {
                    const double q = xg_distance(xr[R], yr[R], xc[C + u], yc[C + u], metric) / p.beta;
                    v[u] = q == 0.0 ? p.sigma2 + p.nugget : xg_tab_eval(tab, q, p.nu, p.con);
                } else {
                    v[u] = (identity_pad && R == C + u) ? 1.0 : 0.0;
                }
            }
        }
        *reinterpret_cast<double2 *>(tile + (long long)r * ts + c) = make_double2(v[0], v[1]);
    }
}

/* Persistent: each CTA a contiguous range of strips, the tables staged once. */
template <bool BIV>
__global__ void __launch_bounds__(XG_GT_THREADS)
    xg_gen_tab_kernel(XgTileArgs T, const int2 *__restrict__ tile_ij, long long units, const double *__restrict__ xr,
                      const double *__restrict__ yr, const double *__restrict__ xc, const double *__restrict__ yc,
                      int n_rows, int n_cols, XgMaternParams p, int metric, int identity_pad,
                      const double *__restrict__ gtab)
{
    extern __shared__ __align__(16) double xg_smem_d[];
    xg_tab_stage(xg_smem_d, gtab, (BIV ? 3 : 1) * XG_TAB_SIZE);
    __syncthreads();
    const int strips = T.ts / XG_GT_ROWS;
    const long long u1 = units * (blockIdx.x + 1LL) / gridDim.x;
    for (long long u = units * blockIdx.x / gridDim.x; u < u1; ++u) {
        const long long t = u / strips;
        xg_gen_tab_strip<BIV>(T.data + t * (long long)T.ts * T.ts, T.ts, tile_ij[t], (int)(u - t * strips), xr, yr, xc,
                              yc, n_rows, n_cols, p, metric, identity_pad, xg_smem_d);
    }
}

/* closed forms of half-integer order and orders beyond the table, for a batch */
__device__ __noinline__ void xg_gen_direct_strip(double *tile, int ts, int2 ij, int strip,
                                                    const double *__restrict__ x, const double *__restrict__ y, int n,
                                                    const XgMaternParams &p, int metric)
{
    for (int e = (int)threadIdx.x; e < XG_GT_ROWS * ts; e += XG_GT_THREADS) {
        const int rr = e / ts, c = e - rr * ts, r = strip * XG_GT_ROWS + rr;
        const int R = ij.x * ts + r, C = ij.y * ts + c;
        tile[(long long)r * ts + c] = R < n && C < n ? xg_matern_value(xg_distance(x[R], y[R], x[C], y[C], metric), p)
                                                     : (R == C ? 1.0 : 0.0);
    }
}

/* every field of a batch: the strips of all fields in one list (S.blk_start),
 * a CTA's range restaging the table where a new field begins */
__global__ void __launch_bounds__(XG_GT_THREADS, 3)
    xg_gen_tab_batch_kernel(XgTileArgs base, const XgBField *__restrict__ F, XgBStep S, long long units,
                            const double *__restrict__ x, const double *__restrict__ y, int metric,
                            const double *__restrict__ gtab)
{
    extern __shared__ __align__(16) double xg_smem_d[];
    __shared__ XgMaternParams p; /* the field's, restaged with its table */
    const int strips = base.ts / XG_GT_ROWS;
    const long long u1 = units * (blockIdx.x + 1LL) / gridDim.x;
    int field = -1;
    for (long long u = units * blockIdx.x / gridDim.x; u < u1;) {
        long long local;
        const int f = xg_batch_resolve(S, u, &local);
        const XgBField &fd = F[f];
        const bool tabbed = xg_tab_wanted(fd.p, fd.N);
        if (f != field) {
            __syncthreads();
            if (tabbed) xg_tab_stage(xg_smem_d, gtab + (long long)f * XG_TAB_SIZE, XG_TAB_SIZE);
            if (threadIdx.x == 0) p = fd.p;
            __syncthreads();
            field = f;
        }
        const double *xf = x + fd.vec_off, *yf = y + fd.vec_off;
        const long long n = xg_num_lower_tiles(fd.nt) * strips;
        for (; u < u1 && local < n; ++u, ++local) {
            const long long t = local / strips;
            double *tile = base.data + (fd.tile_off + t) * (long long)base.ts * base.ts;
            const int2 ij = xg_tile_decode_fast(t, fd.nt);
            const int strip = (int)(local - t * strips);
            if (tabbed)
                xg_gen_tab_strip<false>(tile, base.ts, ij, strip, xf, yf, xf, yf, fd.N, fd.N, p, metric, 1, xg_smem_d);
            else
                xg_gen_direct_strip(tile, base.ts, ij, strip, xf, yf, fd.N, p, metric);
        }
    }
}

/* ========================================================================== */
/* gradient contraction and derivative tiles                                  */
/* ========================================================================== */

__device__ __noinline__ void xg_grad_tab_rare(double r, const XgTabFns &P, double *g)
{
    double m;
    xg_matern_grad(r, P.f[0].nu, P.f[0].con, P.sigma2, P.beta, P.dlogcon, &m, g, g + 1, g + 2);
}

/* sum over the lower triangle of W_RC (dSigma/dtheta_p)_RC, W = (alpha alpha^T - S) / 2
 * doubled off the diagonal, as xg_grad_contract_kernel: each CTA a contiguous
 * range of 8-row strips of the lower tiles of S; partial sums of the four
 * parameters to part[4 blockIdx.x + p] */
__global__ void __launch_bounds__(XG_GT_THREADS)
    xg_grad_contract_tab_kernel(const double *__restrict__ S, int nt, int ts, long long units,
                                const double *__restrict__ x, const double *__restrict__ y,
                                const double *__restrict__ alpha, int N, XgTabFns P, int nugget, int metric,
                                const double *__restrict__ gtab, double *__restrict__ part)
{
    extern __shared__ __align__(16) double xg_smem_d[];
    __shared__ double red[4][XG_GT_THREADS / 32];
    xg_tab_stage(xg_smem_d, gtab, 3 * XG_TAB_SIZE);
    __syncthreads();
    const int strips = ts / XG_GT_ROWS, half = ts / 2;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    const long long u1 = units * (blockIdx.x + 1LL) / gridDim.x;
    for (long long u = units * blockIdx.x / gridDim.x; u < u1; ++u) {
        const long long t = u / strips;
        const int2 ij = xg_tile_decode_fast(t, nt);
        const double *tile = S + t * (long long)ts * ts;
        const int row0 = (int)(u - t * strips) * XG_GT_ROWS;
        for (int e = (int)threadIdx.x; e < XG_GT_ROWS * half; e += XG_GT_THREADS) {
            const int rr = e / half, c = 2 * (e - rr * half), r = row0 + rr;
            const int R = ij.x * ts + r, C = ij.y * ts + c;
            if (R >= N || C > R) continue;
            const double xr = x[R], yr = y[R], ar = alpha[R];
            const double2 s2 = *reinterpret_cast<const double2 *>(tile + (long long)r * ts + c);
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                const int Cc = C + v;
                if (Cc > R) continue;
                const double w = (Cc == R ? 0.5 : 1.0) * (ar * alpha[Cc] - (v ? s2.y : s2.x));
                const double q = xg_distance(xr, yr, x[Cc], y[Cc], metric) / P.beta;
                if (q == 0.0) {
                    acc[0] += w;              /* dSigma/dsigma2 = 1 on the zero-distance branch */
                    if (nugget) acc[3] += w;  /* dSigma/dtau2 */
                    continue;
                }
                const unsigned i = xg_tab_index(q);
                if (i < XG_TAB_NINT) {
                    const double d = q - xg_tab_centre(q), we = w * exp(-q);
                    acc[0] = fma(we, xg_tab_poly(xg_smem_d, i, d), acc[0]);
                    acc[1] = fma(we, xg_tab_poly(xg_smem_d + XG_TAB_SIZE, i, d), acc[1]);
                    acc[2] = fma(we, xg_tab_poly(xg_smem_d + 2 * XG_TAB_SIZE, i, d), acc[2]);
                } else {
                    double g[3];
                    xg_grad_tab_rare(q, P, g);
                    for (int m = 0; m < 3; ++m) acc[m] += w * g[m];
                }
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
        for (int w = 0; w < XG_GT_THREADS / 32; ++w) v += red[threadIdx.x][w];
        part[4 * (long long)blockIdx.x + threadIdx.x] = v;
    }
}

/* dSigma/dtheta_which into full nt x nt tiles, as xg_dsigma_full_kernel */
__global__ void __launch_bounds__(XG_GT_THREADS)
    xg_dsigma_full_tab_kernel(double *__restrict__ D, int nt, int ts, long long units, const double *__restrict__ x,
                              const double *__restrict__ y, int N, XgTabFns P, int metric, int which,
                              const double *__restrict__ gtab)
{
    extern __shared__ __align__(16) double xg_smem_d[];
    xg_tab_stage(xg_smem_d, gtab + (long long)which * XG_TAB_SIZE, XG_TAB_SIZE);
    __syncthreads();
    const int strips = ts / XG_GT_ROWS, half = ts / 2;
    const long long u1 = units * (blockIdx.x + 1LL) / gridDim.x;
    for (long long u = units * blockIdx.x / gridDim.x; u < u1; ++u) {
        const long long slot = u / strips;
        const int B = (int)(slot / nt), A = (int)(slot - (long long)B * nt);
        double *tile = D + slot * (long long)ts * ts;
        const int row0 = (int)(u - slot * strips) * XG_GT_ROWS;
        for (int e = (int)threadIdx.x; e < XG_GT_ROWS * half; e += XG_GT_THREADS) {
            const int rr = e / half, c = 2 * (e - rr * half), r = row0 + rr;
            const int ga = A * ts + r, gb = B * ts + c;
            double v[2] = {0.0, 0.0};
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                if (ga >= N || gb + m >= N) continue;
                const double q = xg_distance(x[ga], y[ga], x[gb + m], y[gb + m], metric) / P.beta;
                const unsigned i = xg_tab_index(q);
                if (q == 0.0) {
                    v[m] = 0.0;
                } else if (i < XG_TAB_NINT) {
                    v[m] = xg_tab_poly(xg_smem_d, i, q - xg_tab_centre(q)) * exp(-q);
                } else {
                    double g[3];
                    xg_grad_tab_rare(q, P, g);
                    v[m] = which == 0 ? g[0] : which == 1 ? g[1] : g[2];
                }
            }
            *reinterpret_cast<double2 *>(tile + (long long)r * ts + c) = make_double2(v[0], v[1]);
        }
    }
}

/* ========================================================================== */
/* launchers                                                                  */
/* ========================================================================== */

static int g_tab_sms = 148;

cudaError_t xg_tab_kernels_configure(int sm_count)
{
    g_tab_sms = sm_count;
    const int three = 3 * XG_TAB_SIZE * (int)sizeof(double);
    cudaError_t e = cudaFuncSetAttribute(xg_gen_tab_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, three);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(xg_grad_contract_tab_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, three);
    return e;
}

size_t xg_tab_doubles() { return 3 * (size_t)XG_TAB_SIZE; }

static unsigned xg_tab_grid(long long units, int per_sm)
{
    const long long g = (long long)g_tab_sms * per_sm;
    return (unsigned)(units < g ? units : g);
}

bool xg_tab_covers(const XgMaternParams &p, int n)
{
    if (n < XG_TAB_MIN_N || !(p.nu <= XG_TAB_NU) || !xg_tab_scale_ok(p.con)) return false;
    if (p.bivariate)
        return p.nu2 <= XG_TAB_NU && p.nu12 <= XG_TAB_NU && xg_tab_scale_ok(p.con2) && xg_tab_scale_ok(p.con12);
    return xg_tab_scale_ok(p.con / p.beta); /* of the derivatives; the covariance follows the same rule */
}

void xg_launch_gen_tab(const XgTileArgs &T, const int2 *tile_ij, long long ntiles, const double *xr, const double *yr,
                       const double *xc, const double *yc, int n_rows, int n_cols, const XgMaternParams &p, int metric,
                       int identity_pad, double *tab, cudaStream_t st)
{
    XgTabFns P = {};
    P.f[0].nu = p.nu;
    P.f[0].con = p.con;
    P.f[0].tm = p.tm;
    if (p.bivariate) {
        P.f[1].nu = p.nu2;
        P.f[1].con = p.con2;
        P.f[1].tm = xg_temme_consts(p.nu2);
        P.f[2].nu = p.nu12;
        P.f[2].con = p.con12;
        P.f[2].tm = xg_temme_consts(p.nu12);
    }
    xg_tab_build_kernel<false><<<dim3(XG_TAB_BUILD_BLOCKS, p.bivariate ? 3 : 1), 64, 0, st>>>(tab, P);
    const long long units = ntiles * (T.ts / XG_GT_ROWS);
    if (p.bivariate)
        xg_gen_tab_kernel<true><<<xg_tab_grid(units, 2), XG_GT_THREADS, 3 * XG_TAB_SIZE * sizeof(double), st>>>(
            T, tile_ij, units, xr, yr, xc, yc, n_rows, n_cols, p, metric, identity_pad, tab);
    else
        xg_gen_tab_kernel<false><<<xg_tab_grid(units, 6), XG_GT_THREADS, XG_TAB_SIZE * sizeof(double), st>>>(
            T, tile_ij, units, xr, yr, xc, yc, n_rows, n_cols, p, metric, identity_pad, tab);
}

void xg_launch_batch_gen(const XgTileArgs &base, const XgBField *F, int nfields, const XgBStep &S, long long blocks,
                         const double *x, const double *y, int metric, double *tab, cudaStream_t st)
{
    if (blocks <= 0) return;
    xg_tab_build_batch_kernel<<<dim3(XG_TAB_BUILD_BLOCKS, nfields < 65535 ? nfields : 65535), 64, 0, st>>>(tab, F,
                                                                                                         nfields);
    xg_gen_tab_batch_kernel<<<xg_tab_grid(blocks, 6), XG_GT_THREADS, XG_TAB_SIZE * sizeof(double), st>>>(
        base, F, S, blocks, x, y, metric, tab);
}

static XgTabFns xg_tab_grad_fns(const XgMaternParams &p, double dlogcon)
{
    XgTabFns P = {};
    P.f[0].nu = p.nu;
    P.f[0].con = p.con;
    P.sigma2 = p.sigma2;
    P.beta = p.beta;
    P.dlogcon = dlogcon;
    return P;
}

void xg_launch_grad_tables(const XgMaternParams &p, double dlogcon, double *tab, cudaStream_t st)
{
    xg_tab_build_kernel<true><<<dim3(XG_TAB_BUILD_BLOCKS, 1), 64, 0, st>>>(tab, xg_tab_grad_fns(p, dlogcon));
}

long long xg_grad_contract_tab_blocks(long long ntiles, int ts)
{
    return xg_tab_grid(ntiles * (ts / XG_GT_ROWS), 2);
}

void xg_launch_grad_contract_tab(const double *S, long long ntiles, int nt, int ts, const double *x, const double *y,
                                 const double *alpha, int N, const XgMaternParams &p, int kernel, int metric,
                                 double dlogcon, const double *tab, double *part, cudaStream_t st)
{
    xg_grad_contract_tab_kernel<<<(unsigned)xg_grad_contract_tab_blocks(ntiles, ts), XG_GT_THREADS,
                                  3 * XG_TAB_SIZE * sizeof(double), st>>>(
        S, nt, ts, ntiles * (ts / XG_GT_ROWS), x, y, alpha, N, xg_tab_grad_fns(p, dlogcon), kernel == 1, metric, tab,
        part);
}

void xg_launch_dsigma_full_tab(double *D, int nt, int ts, const double *x, const double *y, int N,
                               const XgMaternParams &p, double dlogcon, int metric, int which, const double *tab,
                               cudaStream_t st)
{
    const long long units = (long long)nt * nt * (ts / XG_GT_ROWS);
    xg_dsigma_full_tab_kernel<<<xg_tab_grid(units, 6), XG_GT_THREADS, XG_TAB_SIZE * sizeof(double), st>>>(
        D, nt, ts, units, x, y, N, xg_tab_grad_fns(p, dlogcon), metric, which, tab);
}
