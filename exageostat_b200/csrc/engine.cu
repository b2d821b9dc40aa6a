/*
 * Host engine behind the reference C API (capi.cpp).
 *
 * One process-wide context (exageostat_init) owns the CUDA stream.  Each
 * MLE_data owns one XgField (stored in data->descC): the device locations,
 * z, the lower-tile covariance / factor and the solve buffers.  An
 * evaluation is a fixed launch sequence on the context stream:
 *
 *   generate Sigma(theta) tiles -> for k: POTRF(k,k) [+ log-det, + z block
 *   solve] -> TRSM panel k [+ z update] -> trailing update k -> finalize
 *
 * and one device-to-host copy of the result.  Nothing here calls exit().
 */
#include <math.h>
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <sys/time.h>

#include <algorithm>
#include <condition_variable>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/exageostat_b200.h"
#include "kbessel.cuh"
#include "xg_common.cuh"
#include "xg_engine.h"
#include "xg_kernels.h"

/* ------------------------------------------------------------------------- */
/* errors                                                                    */
/* ------------------------------------------------------------------------- */

static thread_local std::string g_last_error;

int xg_fail(int code, const char *fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_last_error = buf;
    return code;
}

static int xg_cuda_fail(cudaError_t e, const char *what)
{
    return xg_fail(XG_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

#define XG_CU(call)                                                                                                    \
    do {                                                                                                               \
        cudaError_t _e = (call);                                                                                       \
        if (_e != cudaSuccess) return xg_cuda_fail(_e, #call);                                                         \
    } while (0)

extern "C" const char *exageostat_last_error(void) { return g_last_error.c_str(); }

/* ------------------------------------------------------------------------- */
/* context                                                                   */
/* ------------------------------------------------------------------------- */

XgContext g_xg;

typedef CUresult (*XgEncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                     const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                     CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static XgEncodeTiledFn g_encode = nullptr;

int xg_context_start(int dts)
{
    std::lock_guard<std::mutex> lk(g_xg.mu);
    if (g_xg.initialized) return XG_OK;
    int dev = 0;
    XG_CU(cudaGetDevice(&dev));
    cudaDeviceProp prop;
    XG_CU(cudaGetDeviceProperties(&prop, dev));
    if (prop.major != 10)
        return xg_fail(XG_ERR_UNSUPPORTED, "device %d (%s, sm_%d%d) is not a B200-class sm_100 GPU", dev, prop.name,
                       prop.major, prop.minor);
    XG_CU(cudaStreamCreateWithFlags(&g_xg.stream, cudaStreamNonBlocking));
    int prio_least = 0, prio_greatest = 0;
    XG_CU(cudaDeviceGetStreamPriorityRange(&prio_least, &prio_greatest));
    XG_CU(cudaStreamCreateWithPriority(&g_xg.stream_hi, cudaStreamNonBlocking, prio_greatest));
    cudaDriverEntryPointQueryResult q;
    void *fn = nullptr;
    XG_CU(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q));
    if (!fn || q != cudaDriverEntryPointSuccess)
        return xg_fail(XG_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    g_encode = (XgEncodeTiledFn)fn;
    cudaError_t e = xg_kernels_configure();
    if (e == cudaSuccess) e = xg_gradient_kernels_configure();
    if (e == cudaSuccess) e = xg_mixed_kernels_configure();
    if (e == cudaSuccess) e = xg_dag_kernels_configure();
    if (e == cudaSuccess) e = xg_rows_kernels_configure();
    if (e == cudaSuccess) e = xg_solve_kernels_configure();
    if (e == cudaSuccess) e = xg_tab_kernels_configure(prop.multiProcessorCount);
    if (e == cudaSuccess) e = xg_sliced_kernels_configure();
    if (e != cudaSuccess) return xg_cuda_fail(e, "kernel attribute setup");
    g_xg.device = dev;
    g_xg.sm_count = prop.multiProcessorCount;
    g_xg.memory = prop.totalGlobalMem;
    g_xg.dts = dts;
    g_xg.initialized = true;
    return XG_OK;
}

int xg_context_require()
{
    if (g_xg.initialized) return XG_OK;
    /* The reference requires exageostat_init first; starting lazily keeps
     * the one-shot entry points usable on their own. */
    return xg_context_start(0);
}

/* tile size: a multiple of 128 in [128, XG_MAX_TS]; 0 picks by problem size */
int xg_choose_ts(int N, int dts)
{
    if (dts <= 0) {
        if (N <= 1024) return 128;
        if (N <= 8192) return 256;
        return 512;
    }
    int ts = ((dts + 127) / 128) * 128;
    if (ts < 128) ts = 128;
    if (ts > XG_MAX_TS) ts = XG_MAX_TS;
    return ts;
}

static bool xg_i8_take_back(bool in_use);
static void xg_i8_free(XgTileMatrix &M);

cudaError_t xg_malloc_bytes(void **p, size_t bytes)
{
    cudaError_t e = cudaMalloc(p, bytes);
    for (int in_use = 0; in_use < 2 && e == cudaErrorMemoryAllocation; ++in_use)
        if (xg_i8_take_back(in_use != 0)) {
            cudaGetLastError();
            e = cudaMalloc(p, bytes);
        }
    if (e != cudaSuccess) {
        cudaGetLastError();
        *p = nullptr;
    }
    return e;
}

cudaError_t xg_alloc_parts(const XgPart *parts, int n, bool take_back)
{
    size_t total = 0;
    for (int i = 0; i < n; ++i) total += (parts[i].bytes + 255) / 256 * 256;
    char *base = nullptr;
    const cudaError_t e = take_back ? xg_malloc(&base, total) : cudaMalloc(&base, total);
    if (e != cudaSuccess) {
        cudaGetLastError();
        base = nullptr;
    }
    for (int i = 0; i < n; ++i) {
        *parts[i].p = base;
        if (base) base += (parts[i].bytes + 255) / 256 * 256;
    }
    return e;
}

/* ------------------------------------------------------------------------- */
/* lower-tile matrices                                                       */
/* ------------------------------------------------------------------------- */

int xg_tm_alloc(XgTileMatrix &M, int N, int ts)
{
    M.N = N;
    M.ts = ts;
    M.nt = (N + ts - 1) / ts;
    M.ntiles = xg_num_lower_tiles(M.nt);
    const size_t elements = (size_t)M.ntiles * ts * ts;
    const int nb = (N + XG_DAG_BLOCK - 1) / XG_DAG_BLOCK;
    const XgPart parts[] = {{&M.d, elements},
                            {&M.dinv, (size_t)M.nt * ts * 32},
                            {&M.tab, xg_tab_doubles()},
                            {&M.ij, (size_t)M.ntiles},
                            {&M.dag, (size_t)(xg_dag_words(nb) + xg_trsv_words(nb))}};
    cudaError_t e = xg_alloc_parts(parts, 5);
    if (e != cudaSuccess)
        return xg_fail(XG_ERR_NO_MEMORY, "cannot allocate %.2f GB for %lld covariance tiles: %s",
                       elements * sizeof(double) / 1e9, M.ntiles, cudaGetErrorString(e));
    int2 *hij = (int2 *)malloc(sizeof(int2) * M.ntiles);
    for (int j = 0; j < M.nt; ++j)
        for (int i = j; i < M.nt; ++i) hij[xg_tile_index(i, j, M.nt)] = make_int2(i, j);
    e = cudaMemcpy(M.ij, hij, sizeof(int2) * M.ntiles, cudaMemcpyHostToDevice);
    free(hij);
    if (e != cudaSuccess) return xg_cuda_fail(e, "tile index table");
    return xg_encode_tiles(&M.map, M.d, M.ntiles, ts);
}

/* TMA view of a lower-tile store: a 2-D FP64 tensor [ntiles * ts rows][ts
 * columns], boxes of 128 rows x 16 columns (128 bytes, swizzled) */
int xg_encode_tiles(CUtensorMap *map, double *base, long long ntiles, int ts)
{
    cuuint64_t dims[2] = {(cuuint64_t)ts, (cuuint64_t)ntiles * ts};
    cuuint64_t strides[1] = {(cuuint64_t)ts * sizeof(double)};
    cuuint32_t box[2] = {16, 128};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, base, dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return xg_fail(XG_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return XG_OK;
}

void xg_tm_free(XgTileMatrix &M)
{
    if (M.d) cudaFree(M.d);
    xg_i8_free(M);
    M.tab = nullptr;
    M.dag = nullptr;
    M.d = nullptr;
    M.ij = nullptr;
    M.dinv = nullptr;
}

XgMaternParams xg_params(const double *theta, int kernel)
{
    XgMaternParams p;
    p.bivariate = 0;
    p.sigma2b = p.nu2 = p.con2 = p.nu12 = p.con12 = p.cross0 = 0.0;
    p.beta2 = p.beta12 = 0.0;
    if (kernel == 3) {
        /* theta = (a_1, a_2, ., ., nu_1, nu_2, ., ., ., ., .): the constants of
         * core_dcmg_bivariate_flexible (core_zcmg.c:1524-1556), in its order;
         * at zero distance the reference stores theta[0], theta[1] and rho
         * (:1565-1568) */
        const double scale1 = theta[0], scale2 = theta[1], nu1 = theta[4], nu2 = theta[5];
        const double scale12 = pow(0.5 * (pow(scale1, -2) + pow(scale2, -2)) + theta[2] * (1 - theta[3]), -0.5);
        const double nu12 = 0.5 * (nu1 + nu2) + theta[6] * (1 - theta[7]);
        const double rho = theta[8] * theta[9] * theta[10] * pow(scale12, 2 * theta[6] + (nu1 + nu2)) *
                           tgamma(0.5 * (nu1 + nu2) + 1) * tgamma(nu12) / tgamma(nu12 + 1);
        const double s11 = theta[8] * theta[8] * pow(scale1, 2 * theta[6] + nu1 + nu1) * tgamma(nu1);
        const double s22 = theta[9] * theta[9] * pow(scale2, 2 * theta[6] + nu2 + nu2) * tgamma(nu2);
        p.bivariate = 1;
        p.sigma2 = theta[0];
        p.sigma2b = theta[1];
        p.cross0 = rho;
        p.beta = scale1;
        p.beta2 = scale2;
        p.beta12 = scale12;
        p.nu = nu1;
        p.nu2 = nu2;
        p.nu12 = nu12;
        p.nugget = 0.0;
        p.half_integer = -1;
        double con1 = pow(2, (nu1 - 1)) * tgamma(nu1);
        con1 = 1.0 / con1;
        p.con = s11 * con1;
        double con2 = pow(2, (nu2 - 1)) * tgamma(nu2);
        con2 = 1.0 / con2;
        p.con2 = s22 * con2;
        double con12 = pow(2, (nu12 - 1)) * tgamma(nu12);
        con12 = 1.0 / con12;
        p.con12 = rho * con12;
        p.tm = xg_temme_consts(nu1);
        return p;
    }
    if (kernel == 2) {
        /* theta = (sigma_1^2, sigma_2^2, beta, nu_1, nu_2, rho): the constants of
         * core_dcmg_bivariate_parsimonious (core_zcmg.c:1637-1651), in its order */
        p.bivariate = 1;
        p.sigma2 = theta[0];
        p.sigma2b = theta[1];
        p.beta = theta[2];
        p.nu = theta[3];
        p.nu2 = theta[4];
        p.nugget = 0.0;
        p.half_integer = -1;
        double con1 = pow(2, (theta[3] - 1)) * tgamma(theta[3]);
        con1 = 1.0 / con1;
        p.con = theta[0] * con1;
        double con2 = pow(2, (theta[4] - 1)) * tgamma(theta[4]);
        con2 = 1.0 / con2;
        p.con2 = theta[1] * con2;
        p.nu12 = 0.5 * (theta[3] + theta[4]);
        const double rho = theta[5] * sqrt((tgamma(theta[3] + 1) * tgamma(theta[4] + 1)) /
                                           (tgamma(theta[3]) * tgamma(theta[4]))) *
                           tgamma(p.nu12) / tgamma(p.nu12 + 1);
        double con12 = pow(2, (p.nu12 - 1)) * tgamma(p.nu12);
        con12 = 1.0 / con12;
        p.con12 = rho * sqrt(theta[0] * theta[1]) * con12;
        p.cross0 = rho * sqrt(theta[0] * theta[1]);
        p.beta2 = p.beta12 = p.beta;
        p.tm = xg_temme_consts(p.nu);
        return p;
    }
    p.sigma2 = theta[0];
    p.beta = theta[1];
    p.nu = theta[2];
    p.nugget = (kernel == 1) ? theta[3] : 0.0;
    /* core_zcmg.c:976-978 */
    double con = pow(2, (theta[2] - 1)) * tgamma(theta[2]);
    con = 1.0 / con;
    p.con = theta[0] * con;
    p.half_integer = (theta[2] == 0.5) ? 0 : (theta[2] == 1.5) ? 1 : (theta[2] == 2.5) ? 2 : -1;
    p.tm = xg_temme_consts(theta[2]);
    return p;
}

int xg_check_theta(const double *theta, int kernel)
{
    if (kernel == 3) {
        for (int i = 0; i < 11; ++i)
            if (!isfinite(theta[i])) return xg_fail(XG_ERR_BAD_ARGUMENT, "theta[%d] is not finite", i);
        const int pos[4] = {0, 1, 4, 5}; /* the two scales and smoothnesses */
        for (int i : pos)
            if (!(theta[i] > 0)) return xg_fail(XG_ERR_BAD_ARGUMENT, "theta[%d] = %g must be positive", i, theta[i]);
        if (theta[4] > 25.0 || theta[5] > 25.0)
            return xg_fail(XG_ERR_BAD_ARGUMENT, "smoothness above the supported maximum 25");
        return XG_OK;
    }
    if (kernel == 2) {
        for (int i = 0; i < 6; ++i)
            if (!isfinite(theta[i])) return xg_fail(XG_ERR_BAD_ARGUMENT, "theta[%d] is not finite", i);
        for (int i = 0; i < 5; ++i)
            if (!(theta[i] > 0)) return xg_fail(XG_ERR_BAD_ARGUMENT, "theta[%d] = %g must be positive", i, theta[i]);
        if (theta[3] > 25.0 || theta[4] > 25.0)
            return xg_fail(XG_ERR_BAD_ARGUMENT, "smoothness above the supported maximum 25");
        return XG_OK;
    }
    const int np = kernel == 1 ? 4 : 3;
    for (int i = 0; i < np; ++i)
        if (!isfinite(theta[i])) return xg_fail(XG_ERR_BAD_ARGUMENT, "theta[%d] is not finite", i);
    if (!(theta[0] > 0) || !(theta[1] > 0) || !(theta[2] > 0))
        return xg_fail(XG_ERR_BAD_ARGUMENT, "theta = (%g, %g, %g) must be positive", theta[0], theta[1], theta[2]);
    if (theta[2] > 25.0)
        return xg_fail(XG_ERR_BAD_ARGUMENT, "smoothness nu = %g is above the supported maximum 25", theta[2]);
    if (kernel == 1 && theta[3] < 0) return xg_fail(XG_ERR_BAD_ARGUMENT, "nugget %g must be >= 0", theta[3]);
    return XG_OK;
}

/* Largest dimension factored by the tile DAG where the INT8 path does not apply.  Milliseconds per evaluation,
 * per-step launches against the DAG: N = 1000 0.73 / 0.45, 3000 2.83 / 1.35,
 * 6000 6.43 / 3.57, 10000 17.9 / 12.8, 14000 38.2 / 32.4, 20000 97.7 / 90.9,
 * 26000 192.3 / 196.1, 32000 352 / 358: past about 22000 the trailing updates
 * fill the chip by themselves and the operands of the DAG's tasks, spread over
 * many columns, no longer stay in L2. */
#define XG_DAG_MAX_N 22000

static int xg_factor_sliced(XgTileMatrix &M, XgSliced *sl, double *v, double *part, int *status,
                            const XgFactorStreams &fs);
static bool xg_i8_acquire(XgTileMatrix &M);
static bool xg_i8_acquire_inverse(XgTileMatrix &M);

/* Block columns J0 .. J1 - 1 of M by the tile DAG: the whole factorisation
 * (0, nb), or one window of it (words: its next-task word; the flags of the
 * whole matrix were cleared when the factorisation began). */
static void xg_launch_dag_columns(XgTileMatrix &M, int J0, int J1, int *next, double *v, double *part, int *status,
                                  int ctas, cudaStream_t st)
{
    const int nb = (M.N + XG_DAG_BLOCK - 1) / XG_DAG_BLOCK;
    if (J1 > nb) J1 = nb;
    XgDag G = {};
    G.data = M.d;
    G.ts = M.ts;
    G.one.nt = M.nt;
    G.one.nb = nb;
    G.J0 = J0;
    G.ntasks = xg_num_lower_tiles(nb - J0) - xg_num_lower_tiles(nb - J1);
    G.next = (unsigned *)next;
    G.abort = M.dag + 1;
    G.flags = M.dag + 2;
    G.dinv = M.dinv;
    G.v = v;
    G.part = part;
    G.status = status;
    xg_launch_dag(M.map, G, ctas, st);
}

/* Smallest dimension whose FP64 factorisation runs its updates on the INT8
 * tensor cores (seven digits, sliced.cu) instead of DMMA, by tile size: a
 * panel is one chunk of the product, and each chunk's sums are brought back
 * and scaled once, so small tiles pay that more often.  Milliseconds, DMMA
 * dataflow / INT8, of a log-likelihood and of a gradient: ts = 512 N = 6000
 * 3.43 / 3.52 and 8.6 / 7.6, 20000 90 / 40 and - / 133; ts = 384 N = 6000 3.44 /
 * 3.51 and 8.6 / 7.7, 7000 5.00 / 4.37 and 12.9 / 10.2; ts = 256 N = 6000 3.43 /
 * 3.78 and 8.6 / 8.2, 7000 4.98 / 4.68 and 12.9 / 10.8, 8100 7.45 / 5.67 and
 * 19.5 / 13.7, 10000 13.3 / 9.0 and 35.2 / 23.0.  At ts = 128
 * the line would be 8500 (12000 21.8 / 16.8), but nothing chooses 128 there
 * (512 takes 11.6), and it is the path that the digits are tested against. */
static int xg_i8_min(int ts) { return ts >= 256 ? 6500 : 1 << 30; }

/* The factorisation of M as one launch of the tile DAG (tile_dag.cu); returns
 * the number of partial sums of either kind. */
static int xg_factor_dag(XgTileMatrix &M, double *v, double *part, int *status, int ctas, cudaStream_t st)
{
    const int nb = (M.N + XG_DAG_BLOCK - 1) / XG_DAG_BLOCK;
    cudaMemsetAsync(M.dag, 0, sizeof(int) * (size_t)xg_dag_words(nb), st);
    xg_launch_dag_columns(M, 0, nb, M.dag, v, part, status, ctas, st);
    return nb;
}

static int xg_digits_alloc(XgDigits &D, const XgTileMatrix &M, int digits);
static void xg_digits_free(XgDigits &D);

/* SMs left free by the persistent trailing-update kernels (one CTA per SM,
 * ~197 KB of shared memory each) while the lookahead panel of the next step
 * (POTRF, TRSM, panel conversion) runs on the high-priority stream: resident
 * CTAs are never preempted, so without free SMs the panel would wait for the
 * whole update. */
#define XG_PANEL_SMS 16

/* Tile columns per group.  One column gives an update 16 (nt - j) jobs of 128
 * x 128, whose last round leaves most of the persistent CTAs idle: counted
 * over the columns 1.7 x the even distribution at 38 tile columns, 1.36 x at
 * 79, 1.24 x at 137; groups of four bring that to 1.21, 1.09 and 1.05, but put
 * three columns' panels between two updates, which the short matrices have
 * nothing to run beside.  Log-likelihood in ms, tiles of 512, K = 4 below:
 *   7 digits   N = 8200  10000  14000  20000  28000  40000
 *     G = 1        6.00   8.80     -    46.6     -    316
 *     G = 2        5.71   7.98   17.9   44.7   109    308
 *     G = 3        6.13   8.17   16.6   42.2   107    305
 *     G = 4        6.52   8.81   17.3   41.1   105    298
 *   4 digits   N = 9000  20000  40000  70000
 *     G = 1        5.00   20.2    117   560
 *     G = 2        5.02   20.1    119   574
 *     G = 3        5.20   21.4    118   573
 * (28 pairs cost an update 2.8 times what ten do, the panels the same: the
 * four-digit form has the panels to hide, not the last rounds.) */
static int xg_sl_group(int nt, int digits)
{
    return digits == 4 ? 1 : nt < 24 ? 2 : nt < 36 ? 3 : 4;
}

static XgSlTask xg_sl_task(int mode, int col, int ncol, int k0, int k1)
{
    XgSlTask S;
    S.mode = mode;
    S.col = col;
    S.ncol = ncol;
    S.k0 = k0;
    S.k1 = k1;
    S.sign = mode == XG_SL_SYRK ? 1.0 : -1.0;
    return S;
}

/* SMs left to the panels of the group that begins at tile column a while U1 of
 * the next group runs on the others.  Per target tile the panels cost the DMMA
 * flops of the TRSM and the group's own chunks, U1 a chunks: sms K / (K + a),
 * clamped to [XG_PANEL_SMS, sms - XG_PANEL_SMS].  K = 4
 * (EXAGEOSTAT_B200_PANEL_K overrides it): seven digits in groups of four at
 * N = 10000 / 20000 / 40000 took 11.0 / 51.4 / 325 ms with K = 1, 9.9 / 46.5 /
 * 317 with 2, 9.2 / 43.8 / 309 with 3, 8.9 / 41.6 / 308 with 4 and 8.6 / 43.6 /
 * 311 with 6; four digits at 20000 / 70000 20.4 / 570 with 4 and 20.9 / 572
 * with 7. */
static int xg_panel_k()
{
    static int v = -1;
    if (v < 0) {
        const char *e = getenv("EXAGEOSTAT_B200_PANEL_K");
        v = e ? atoi(e) : 0;
        if (v < 1 || v > 64) v = 4;
    }
    return v;
}

static int xg_panel_share(int a, int sms)
{
    const int K = xg_panel_k();
    int r = (int)((long long)sms * K / (K + a));
    if (r < XG_PANEL_SMS) r = XG_PANEL_SMS;
    if (r > sms - XG_PANEL_SMS) r = sms - XG_PANEL_SMS;
    return r;
}

/* How the SMs are divided between the panel chain and the split update.
 * "static" (default): the split update runs as a persistent launch on
 * sms - xg_panel_share(a) CTAs, leaving the rest to the panel chain.
 * "dynamic" (EXAGEOSTAT_B200_SL_SHARE=dynamic): both updates launch one CTA
 * per job, so CTAs retire throughout the update and the hardware hands each
 * freed SM to the pending panel kernels first (higher stream priority), the
 * SMs the chain does not need staying with the update. */
static bool xg_sl_dynamic_share()
{
    static int v = -1;
    if (v < 0) {
        const char *e = getenv("EXAGEOSTAT_B200_SL_SHARE");
        v = (e && strcmp(e, "dynamic") == 0) ? 1 : 0;
    }
    return v == 1;
}

/* INT8 tile columns in groups of G = xg_sl_group [a, b), left-looking:
 *   U1     chunks k < a0 (the group before begins at a0) to every target of the group (main stream,
 *          on all but xg_panel_share SMs, beside the panels of the group before)
 *   U2     chunks a0 <= k < a, when those panels are sliced: column a on the panel stream, the
 *          others on the main stream
 *   panel  per column c: chunks a <= k < c (for c > a), then panel(c)
 * update(col, ncol, k0, k1, ctas, stream) and panel(c, stream) do the work.
 * Profiling events (8 per column c, those of the main stream on a group's
 * first column): panel stream before / after the column's updates, after its
 * panel, after slicing (both panel's to record); main stream before / after U1. */
template <class Update, class Panel>
static void xg_sliced_groups(int nt, XgSliced *sl, const XgFactorStreams &fs, Update update, Panel panel)
{
    const bool la = fs.st_hi != nullptr;
    cudaStream_t st = fs.st, sp = la ? fs.st_hi : fs.st;
    auto rec = [&](int k, int e, cudaStream_t s) {
        if (fs.pev) cudaEventRecord(fs.pev[8 * k + e], s);
    };
    const int sms = g_xg.sm_count;
    const int G = xg_sl_group(nt, sl->L.digits);
    const bool dyn = xg_sl_dynamic_share();
    const int all = 1 << 30; /* one CTA per job */
    if (la) {
        cudaEventRecord(sl->ev_a, st); /* the matrix as it comes */
        cudaStreamWaitEvent(sp, sl->ev_a, 0);
    }
    for (int a = 0; a < nt; a += G) {
        const int b = a + G < nt ? a + G : nt, a0 = a - G;
        const int share = dyn ? all : xg_panel_share(a, sms);
        /* main stream: U1 of this group was issued with the group before; U2 of
         * the columns after the first */
        if (la && a > 0) {
            cudaEventRecord(sl->ev_p[0], sp); /* the group before is sliced */
            cudaEventRecord(sl->ev_a, st);    /* U1 of this group is done */
            cudaStreamWaitEvent(st, sl->ev_p[0], 0);
            cudaStreamWaitEvent(sp, sl->ev_a, 0);
        }
        if (a > 0) update(a + 1, b - a - 1, a0, a, sms, st);
        if (la && a > 0) cudaEventRecord(sl->ev_p[1], st);
        rec(a, 4, st);
        const int b1 = b + G < nt ? b + G : nt; /* the next group: chunks k < a */
        update(b, b1 - b, 0, a, !la ? sms : dyn ? all : sms - share, st);
        rec(a, 5, st);
        for (int c = a; c < b; ++c) {
            rec(c, 0, sp);
            if (c == a) {
                /* alone in its group it runs beside U1 of the next column */
                if (a > 0) update(a, 1, a0, a, la && G == 1 ? share : sms, sp);
            } else {
                if (la && a > 0 && c == a + 1) cudaStreamWaitEvent(sp, sl->ev_p[1], 0);
                update(c, 1, a, c, la && b < nt ? share : sms, sp);
            }
            rec(c, 1, sp);
            panel(c, sp);
            rec(c, 3, sp);
            if (c > a) {
                rec(c, 4, st);
                rec(c, 5, st);
            }
            rec(c, 6, st);
            rec(c, 7, st);
        }
    }
    if (la) {
        cudaEventRecord(fs.ev_panel, sp);
        cudaStreamWaitEvent(st, fs.ev_panel, 0);
    }
}

/* X = L^-T by groups of tile columns: the updates from the finished columns
 * (INT8, from the digit planes of X and L); a column's panel is the FP64 block
 * solves with L_bb (one dataflow launch) and its slicing.  Then S = X X^T over
 * the factor in one launch.  Gradients in ms, one column at a time on one
 * stream / in groups beside the panels: seven digits N = 7000 11.1 / 9.7, 10000
 * 22.4 / 20.0, 14000 49.3 / 46.3, 20000 132 / 131, 40000 941 / 942; four digits
 * 9000 11.1 / 10.5, 40000 373 / 364, 70000 1814 / 1793. */
static void xg_inverse_product_sliced(XgTileMatrix &M, XgTileMatrix &X, XgSliced *sl, int *status,
                                      const XgFactorStreams &fs)
{
    const int ts = M.ts, nt = M.nt, bpt = ts / XG_DAG_BLOCK;
    const int nb = (M.N + XG_DAG_BLOCK - 1) / XG_DAG_BLOCK;
    XgTileArgs T{M.d, ts, nt}, TX{X.d, ts, nt};
    const long long plane = (long long)sl->X.plane_rows * ts;
    int *windows = X.dag + xg_dag_words(nb) - nb;
    cudaMemsetAsync(X.dag, 0, sizeof(int) * (size_t)xg_dag_words(nb), fs.st);
    xg_launch_zero_diag(X.d, nt, ts, fs.st);
    XgRowsMaps maps = {};
    maps.y[0] = X.map;
    maps.l[0] = M.map;
    xg_sliced_groups(
        nt, sl, fs,
        [&](int col, int ncol, int k0, int k1, int ctas, cudaStream_t s) {
            if (ncol > 0 && k1 > k0)
                xg_launch_sliced(sl->X, sl->L, TX, xg_sl_task(XG_SL_INVERSE, col, ncol, k0, k1), ctas, status, s);
        },
        [&](int b, cudaStream_t s) {
            const int J0 = b * bpt, J1 = J0 + bpt < nb ? J0 + bpt : nb;
            XgRows G = {};
            G.y[0] = X.d;
            G.dinv[0] = M.dinv;
            G.s = M.d;
            G.ts = ts;
            G.nsys = 1;
            G.J0 = J0;
            G.one.nt = nt;
            G.one.nb = nb;
            G.ntasks = xg_num_lower_tiles(J1) - xg_num_lower_tiles(J0);
            G.next = (unsigned *)(windows + b);
            G.abort = X.dag + 1;
            G.flags = X.dag + 2;
            G.status = status;
            xg_launch_rows(XG_ROWS_INVERSE, maps, G, g_xg.sm_count, s);
            xg_launch_slice_panel(TX, b, 1, sl->X.digits, sl->X.dig, sl->X.scale, plane, status, s);
        });
    xg_launch_sliced(sl->X, sl->X, T, xg_sl_task(XG_SL_SYRK, 0, nt, 0, nt), g_xg.sm_count, status, fs.st);
}

/* X = L^-T, then Sigma^-1 = X X^T over the factor M (lower tiles) */
void xg_inverse_product(XgTileMatrix &M, XgTileMatrix &X, int *status, const XgFactorStreams &fs)
{
    cudaStream_t st = fs.st;
    if (M.i8_factor && M.i8 && xg_i8_acquire_inverse(M)) {
        xg_inverse_product_sliced(M, X, M.i8, status, fs);
        return;
    }
    const int nb = (M.N + XG_DAG_BLOCK - 1) / XG_DAG_BLOCK;
    cudaMemsetAsync(X.dag, 0, sizeof(int) * (size_t)xg_dag_words(nb), st);
    XgRowsMaps maps = {};
    maps.y[0] = X.map;
    maps.l[0] = M.map;
    XgRows G = {};
    G.y[0] = X.d;
    G.dinv[0] = M.dinv;
    G.s = M.d;
    G.ts = M.ts;
    G.nsys = 1;
    G.one.nt = M.nt;
    G.one.nb = nb;
    G.ntasks = 2 * xg_num_lower_tiles(nb);
    G.next = (unsigned *)X.dag;
    G.abort = X.dag + 1;
    G.flags = X.dag + 2;
    G.status = status;
    xg_launch_rows(XG_ROWS_INVERSE, maps, G, g_xg.sm_count, st);
}

/* v <- L^-T v for a factored M */
void xg_solve_transposed(XgTileMatrix &M, double *v, int *status, cudaStream_t st)
{
    const int nb = (M.N + XG_DAG_BLOCK - 1) / XG_DAG_BLOCK;
    int *words = M.dag + xg_dag_words(nb);
    cudaMemsetAsync(words, 0, sizeof(int) * (size_t)xg_trsv_words(nb), st);
    XgTrsv G = {};
    G.data = M.d;
    G.ts = M.ts;
    G.one.nt = M.nt;
    G.one.nb = nb;
    G.ntasks = nb;
    G.next = (unsigned *)words;
    G.abort = words + 1;
    G.flags = words + 2;
    G.dinv = M.dinv;
    G.v = v;
    G.status = status;
    xg_launch_trsv_lower_t(G, g_xg.sm_count, st);
}

/* Cholesky of M in place; with v != nullptr also v <- L^-1 v.  Returns the
 * number n of partial sums of either kind: log-det in part[0:n], |v|^2 in
 * part[n:2n].  Up to XG_DAG_MAX_N one launch of the tile DAG, else a
 * right-looking sequence of launches.  Per step k:
 *   panel   : POTRF(k,k) [+ log-det, + L_kk v_k = v_k]  ->  TRSM(i,k) [+ v_i -= L_ik v_k]
 *   trailing: A_ij -= L_ik L_jk^T, j >= k+1
 * With fs.st_hi the panel of step k+1 runs on the high-priority stream as soon
 * as column k+1 has received the step-k update (the trailing update is split
 * into "column k+1" and "the rest"), so it overlaps the rest of step k.
 * Profiling events (5 per step): panel start, after POTRF, after TRSM,
 * trailing start, trailing end. */
int xg_factor_lookahead(XgTileMatrix &M, double *v, double *part, int *status, int *info, const XgFactorStreams &fs)
{
    /* profiled evaluations keep the per-step launches, whose kernels the profile tells apart */
    M.i8_factor = false;
    if (M.dag && !fs.pev) {
        if (M.N >= xg_i8_min(M.ts) && M.i8_scale && xg_i8_acquire(M)) {
            M.i8_factor = true;
            return xg_factor_sliced(M, M.i8, v, part, status, fs);
        }
        if (M.N <= XG_DAG_MAX_N) return xg_factor_dag(M, v, part, status, g_xg.sm_count, fs.st);
    }
    XgTileArgs T{M.d, M.ts, M.nt};
    const bool la = fs.st_hi != nullptr;
    cudaStream_t sp = la ? fs.st_hi : fs.st; /* panel stream */
    cudaEvent_t *pev = fs.pev;
    const int rhs = v != nullptr;
    if (la) {
        cudaEventRecord(fs.ev_upd, fs.st); /* the generated matrix */
    }
    for (int k = 0; k < M.nt; ++k) {
        if (M.dinv) T.dinv = M.dinv + (size_t)k * M.ts * 32;
        if (la) cudaStreamWaitEvent(sp, fs.ev_upd, 0);
        if (pev) cudaEventRecord(pev[5 * k], sp);
        xg_launch_potrf_tiled(M.map, T, k, v, part, part + M.nt, rhs, status, info, sp);
        if (pev) cudaEventRecord(pev[5 * k + 1], sp);
        if (T.dinv)
            xg_launch_trsm_gemm(M.map, T, k, v, rhs, status, sp);
        else
            xg_launch_trsm_panel(T, k, v, rhs, status, sp);
        if (pev) cudaEventRecord(pev[5 * k + 2], sp);
        if (la) {
            cudaEventRecord(fs.ev_panel, sp);
            cudaStreamWaitEvent(fs.st, fs.ev_panel, 0);
        }
        if (pev) cudaEventRecord(pev[5 * k + 3], fs.st);
        if (k + 1 < M.nt) {
            if (la) {
                xg_launch_syrk_gemm(M.map, T, k, status, fs.st, 1);
                cudaEventRecord(fs.ev_upd, fs.st);
                xg_launch_syrk_gemm(M.map, T, k, status, fs.st, 2);
            } else {
                xg_launch_syrk_gemm(M.map, T, k, status, fs.st, 0);
            }
        }
        if (pev) cudaEventRecord(pev[5 * k + 4], fs.st);
    }
    return M.nt;
}

/* The factorisations of two matrices of one size, without right-hand sides.
 * Up to the INT8 path's sizes they run side by side on half the SMs each: a
 * matrix of 4000 is bound by its chain of diagonal blocks (1.50 ms; its
 * products would take 0.6).  Both, one after the other / side by side in ms: N =
 * 300 0.24 / 0.12, 1000 0.70 / 0.35, 4000 3.00 / 2.04, 9000 13.0 / 12.3.  The
 * launches do not wait on one another. */
void xg_factor_two(XgTileMatrix &A, XgTileMatrix &B, double *part_a, double *part_b, int *status, int *info,
                   const XgFactorStreams &fs)
{
    if (!A.dag || !B.dag || !fs.st_hi || A.N > XG_DAG_MAX_N || A.N >= xg_i8_min(A.ts)) {
        xg_factor_lookahead(A, nullptr, part_a, status, info, fs);
        xg_factor_lookahead(B, nullptr, part_b, status, info, fs);
        return;
    }
    const int half = g_xg.sm_count / 2;
    A.i8_factor = B.i8_factor = false;
    cudaEventRecord(fs.ev_upd, fs.st); /* the generated matrices */
    cudaStreamWaitEvent(fs.st_hi, fs.ev_upd, 0);
    xg_factor_dag(B, nullptr, part_b, status, g_xg.sm_count - half, fs.st_hi);
    xg_factor_dag(A, nullptr, part_a, status, half, fs.st);
    cudaEventRecord(fs.ev_panel, fs.st_hi);
    cudaStreamWaitEvent(fs.st, fs.ev_panel, 0);
}

int xg_factor(XgTileMatrix &M, double *v, double *part, int *status, int *info, cudaStream_t st, cudaEvent_t *pev)
{
    XgFactorStreams fs;
    fs.st = st;
    fs.pev = pev;
    return xg_factor_lookahead(M, v, part, status, info, fs);
}

/* Algorithmic flops of the trailing update after step k: a GEMM (2 ts^3) per
 * off-diagonal tile pair and a SYRK (ts^2 (ts + 1)) per diagonal tile. */
double xg_trailing_flops(int nt, int ts, int k)
{
    const double n = nt - k - 1;
    const double t = ts;
    return n * (n - 1) / 2 * 2 * t * t * t + n * t * t * (t + 1);
}

int xg_field_set_profiling(XgField *f, int on)
{
    if (on && !f->pev) {
        const int n = 8 * f->C.nt;
        f->pev = (cudaEvent_t *)calloc(n, sizeof(cudaEvent_t));
        for (int i = 0; i < n; ++i)
            if (cudaEventCreate(&f->pev[i]) != cudaSuccess) return xg_fail(XG_ERR_CUDA, "profiling events");
    }
    f->profiling = on != 0;
    for (int i = 0; i < 12; ++i) f->prof[i] = 0;
    return XG_OK;
}

static void xg_field_collect_profile(XgField *f)
{
    float ms = 0;
    const int nt = f->C.nt;
    cudaEventElapsedTime(&ms, f->ev[0], f->ev[1]);
    f->prof[0] += ms * 1e-3;
    for (int k = 0; k < nt; ++k) {
        cudaEventElapsedTime(&ms, f->pev[5 * k], f->pev[5 * k + 1]);
        f->prof[1] += ms * 1e-3;
        cudaEventElapsedTime(&ms, f->pev[5 * k + 1], f->pev[5 * k + 2]);
        f->prof[2] += ms * 1e-3;
        if (k + 1 < nt) {
            cudaEventElapsedTime(&ms, f->pev[5 * k + 3], f->pev[5 * k + 4]);
            f->prof[3] += ms * 1e-3;
            f->prof[4] += xg_trailing_flops(nt, f->C.ts, k);
        }
    }
    cudaEventElapsedTime(&ms, f->ev[0], f->ev[2]);
    f->prof[7] += ms * 1e-3;
    /* launches: generation, the sub-block POTRF sequence per step, TRSM and two
     * trailing launches per step but the last (the first trailing launch of
     * the last step but one covers one column and the second is empty),
     * finalize */
    double launches = 1 + (double)nt * xg_potrf_tiled_launches(f->C.ts) + 1;
    for (int k = 0; k + 1 < nt; ++k) launches += 1 + 1 + (k + 2 < nt ? 1 : 0);
    f->prof[5] += launches;
    f->prof[6] += 1;
}

int xg_field_set_data(XgField *f, const double *x, const double *y, const double *z)
{
    cudaStream_t st = g_xg.stream;
    const int nloc = xg_bivariate(f->kernel) ? f->N / 2 : f->N; /* bivariate: two variables per location */
    if (x) XG_CU(cudaMemcpyAsync(f->x, x, nloc * sizeof(double), cudaMemcpyHostToDevice, st));
    if (y) XG_CU(cudaMemcpyAsync(f->y, y, nloc * sizeof(double), cudaMemcpyHostToDevice, st));
    if (z) XG_CU(cudaMemcpyAsync(f->z, z, f->N * sizeof(double), cudaMemcpyHostToDevice, st));
    XG_CU(cudaStreamSynchronize(st));
    if (z) f->have_z = true;
    return XG_OK;
}

/* ------------------------------------------------------------------------- */
/* fields                                                                    */
/* ------------------------------------------------------------------------- */

static int xg_dev_alloc(double **p, size_t n)
{
    cudaError_t e = xg_malloc(p, n * sizeof(double));
    if (e != cudaSuccess) return xg_fail(XG_ERR_NO_MEMORY, "cudaMalloc(%zu doubles): %s", n, cudaGetErrorString(e));
    return cudaMemset(*p, 0, n * sizeof(double)) == cudaSuccess ? XG_OK : XG_ERR_CUDA;
}

void xg_field_destroy(XgField *f)
{
    if (!f) return;
    xg_tm_free(f->C);
    double *bufs[] = {f->x, f->y, f->z, f->v, f->e, f->part, f->out};
    for (double *b : bufs)
        if (b) cudaFree(b);
    if (f->status) cudaFree(f->status);
    if (f->h_out) cudaFreeHost(f->h_out);
    if (f->pev) {
        for (int i = 0; i < 8 * f->C.nt; ++i)
            if (f->pev[i]) cudaEventDestroy(f->pev[i]);
        free(f->pev);
    }
    if (f->ev_panel) cudaEventDestroy(f->ev_panel);
    if (f->ev_upd) cudaEventDestroy(f->ev_upd);
    xg_tm_free(f->X);
    if (f->mx) xg_mixed_destroy(f->mx);
    if (f->sl) xg_sliced_destroy(f->sl);
    if (f->gpart) cudaFree(f->gpart);
    if (f->gout) cudaFree(f->gout);
    for (int i = 0; i < 4; ++i)
        if (f->ev[i]) cudaEventDestroy(f->ev[i]);
    delete f;
}

int xg_field_create(XgField **out, int N, int ts, const double *x, const double *y, int kernel, int metric)
{
    *out = nullptr;
    int rc = xg_context_require();
    if (rc) return rc;
    if (N <= 0) return xg_fail(XG_ERR_BAD_ARGUMENT, "N = %d must be positive", N);
    if (!x || !y) return xg_fail(XG_ERR_BAD_ARGUMENT, "locations are NULL");
    if (xg_bivariate(kernel) && (N & 1))
        return xg_fail(XG_ERR_BAD_ARGUMENT, "bivariate kernel: N = %d must be 2 x the number of locations", N);
    /* bivariate: N / 2 locations, two variables each */
    const int nloc = xg_bivariate(kernel) ? N / 2 : N;
    XgField *f = new XgField();
    f->N = N;
    f->kernel = kernel;
    f->metric = metric;
    rc = xg_tm_alloc(f->C, N, xg_choose_ts(N, ts));
    const size_t Np = (size_t)f->C.nt * f->C.ts;
    if (!rc) rc = xg_dev_alloc(&f->x, Np);
    if (!rc) rc = xg_dev_alloc(&f->y, Np);
    if (!rc) rc = xg_dev_alloc(&f->z, Np);
    if (!rc) rc = xg_dev_alloc(&f->v, Np);
    if (!rc) rc = xg_dev_alloc(&f->e, Np);
    if (!rc) rc = xg_dev_alloc(&f->part, 2 * Np / XG_DAG_BLOCK);
    if (!rc) rc = xg_dev_alloc(&f->out, 8);
    if (!rc && xg_malloc(&f->status, 2 * sizeof(int)) != cudaSuccess) rc = xg_fail(XG_ERR_NO_MEMORY, "status word");
    if (!rc && cudaMallocHost(&f->h_out, 8 * sizeof(double)) != cudaSuccess)
        rc = xg_fail(XG_ERR_NO_MEMORY, "pinned result buffer");
    for (int i = 0; i < 4 && !rc; ++i)
        if (cudaEventCreate(&f->ev[i]) != cudaSuccess) rc = xg_fail(XG_ERR_CUDA, "event");
    if (!rc && (cudaEventCreateWithFlags(&f->ev_panel, cudaEventDisableTiming) != cudaSuccess ||
                cudaEventCreateWithFlags(&f->ev_upd, cudaEventDisableTiming) != cudaSuccess))
        rc = xg_fail(XG_ERR_CUDA, "lookahead events");
    if (!rc && cudaMemcpy(f->x, x, nloc * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess)
        rc = xg_fail(XG_ERR_CUDA, "upload x");
    if (!rc && cudaMemcpy(f->y, y, nloc * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess)
        rc = xg_fail(XG_ERR_CUDA, "upload y");
    if (rc) {
        xg_field_destroy(f);
        return rc;
    }
    f->info = f->status + 1;
    *out = f;
    return XG_OK;
}

int xg_field_set_z(XgField *f, const double *z)
{
    cudaStream_t st = g_xg.stream;
    XG_CU(cudaMemcpyAsync(f->z, z, f->N * sizeof(double), cudaMemcpyHostToDevice, st));
    XG_CU(cudaStreamSynchronize(st));
    f->have_z = true;
    return XG_OK;
}

static int xg_read_status(XgField *f)
{
    const int st = (int)f->h_out[3];
    if (st & XG_ST_NOT_SPD)
        return xg_fail(XG_ERR_NOT_SPD, "the covariance is not positive definite (pivot %d)", (int)f->h_out[4]);
    if (st & XG_ST_TIMEOUT) return xg_fail(XG_ERR_TIMEOUT, "a device pipeline wait timed out");
    if (st) return xg_fail(XG_ERR_CUDA, "device status word 0x%x", st);
    return XG_OK;
}

/* log-likelihood at theta; res[0..2] = loglik, logdet, dotp; times[0..1] =
 * generation and factorisation+solve seconds (CUDA events). */
int xg_field_loglik(XgField *f, const double *theta, double *res, double *times)
{
    int rc = xg_check_theta(theta, f->kernel);
    if (rc) return rc;
    if (!f->have_z) return xg_fail(XG_ERR_BAD_ARGUMENT, "no observations: call MLE_zvg or set z first");
    cudaStream_t st = g_xg.stream;
    XgTileArgs T{f->C.d, f->C.ts, f->C.nt};
    const XgMaternParams p = xg_params(theta, f->kernel);
    XgI8Use use(f->C, p);
    const size_t Np = (size_t)f->C.nt * f->C.ts;
    XG_CU(cudaMemsetAsync(f->status, 0, 2 * sizeof(int), st));
    XG_CU(cudaMemcpyAsync(f->v, f->z, Np * sizeof(double), cudaMemcpyDeviceToDevice, st));
    XG_CU(cudaEventRecord(f->ev[0], st));
    xg_launch_gen(T, f->C.ij, f->C.ntiles, f->x, f->y, f->x, f->y, f->N, f->N, p, f->metric, 1, f->C.tab, st);
    XG_CU(cudaEventRecord(f->ev[1], st));
    XgFactorStreams fs;
    fs.st = st;
    fs.st_hi = g_xg.stream_hi;
    fs.ev_panel = f->ev_panel;
    fs.ev_upd = f->ev_upd;
    fs.pev = f->profiling ? f->pev : nullptr;
    const int np = xg_factor_lookahead(f->C, f->v, f->part, f->status, f->info, fs);
    xg_launch_finalize(f->part, f->part + np, np, f->N, f->out, f->status, f->info, st);
    XG_CU(cudaEventRecord(f->ev[2], st));
    XG_CU(cudaMemcpyAsync(f->h_out, f->out, 5 * sizeof(double), cudaMemcpyDeviceToHost, st));
    XG_CU(cudaGetLastError());
    XG_CU(cudaStreamSynchronize(st));
    if (times) {
        float a = 0, b = 0;
        cudaEventElapsedTime(&a, f->ev[0], f->ev[1]);
        cudaEventElapsedTime(&b, f->ev[1], f->ev[2]);
        times[0] = a * 1e-3;
        times[1] = b * 1e-3;
    }
    if (f->profiling) xg_field_collect_profile(f);
    rc = xg_read_status(f);
    if (rc) return rc;
    res[0] = f->h_out[0];
    res[1] = f->h_out[1];
    res[2] = f->h_out[2];
    return XG_OK;
}

/* z = chol(Sigma(theta)) e, e = nrand (N host doubles) */
int xg_field_zvg(XgField *f, const double *theta, const double *nrand, double *times)
{
    int rc = xg_check_theta(theta, f->kernel);
    if (rc) return rc;
    cudaStream_t st = g_xg.stream;
    XgTileArgs T{f->C.d, f->C.ts, f->C.nt};
    const XgMaternParams p = xg_params(theta, f->kernel);
    XgI8Use use(f->C, p);
    XG_CU(cudaMemsetAsync(f->status, 0, 2 * sizeof(int), st));
    XG_CU(cudaMemcpyAsync(f->e, nrand, f->N * sizeof(double), cudaMemcpyHostToDevice, st));
    XG_CU(cudaEventRecord(f->ev[0], st));
    xg_launch_gen(T, f->C.ij, f->C.ntiles, f->x, f->y, f->x, f->y, f->N, f->N, p, f->metric, 1, f->C.tab, st);
    XG_CU(cudaEventRecord(f->ev[1], st));
    XgFactorStreams fs;
    fs.st = st;
    fs.st_hi = g_xg.stream_hi;
    fs.ev_panel = f->ev_panel;
    fs.ev_upd = f->ev_upd;
    xg_factor_lookahead(f->C, nullptr, f->part, f->status, f->info, fs);
    xg_launch_trmv_lower(T, f->e, f->z, f->status, st);
    XG_CU(cudaEventRecord(f->ev[2], st));
    XG_CU(cudaGetLastError());
    XG_CU(cudaStreamSynchronize(st));
    /* status and info are ints on the device: widen them into the slots
     * xg_read_status reads */
    int sv[2];
    XG_CU(cudaMemcpy(sv, f->status, sizeof sv, cudaMemcpyDeviceToHost));
    f->h_out[3] = sv[0];
    f->h_out[4] = sv[1];
    if (times) {
        float a = 0, b = 0;
        cudaEventElapsedTime(&a, f->ev[0], f->ev[1]);
        cudaEventElapsedTime(&b, f->ev[1], f->ev[2]);
        times[0] = a * 1e-3;
        times[1] = b * 1e-3;
    }
    rc = xg_read_status(f);
    if (rc) return rc;
    f->have_z = true;
    return XG_OK;
}

/* digamma: upward recurrence to x >= 10, then the asymptotic series
 * psi(x) = ln x - 1/(2x) - sum_k B_2k / (2k x^2k) (Abramowitz & Stegun 6.3.18) */
double xg_digamma(double x)
{
    double r = 0.0;
    while (x < 10.0) {
        r -= 1.0 / x;
        x += 1.0;
    }
    const double i2 = 1.0 / (x * x);
    const double series =
        i2 * (1.0 / 12 - i2 * (1.0 / 120 - i2 * (1.0 / 252 - i2 * (1.0 / 240 - i2 * (1.0 / 132 - i2 * (691.0 / 32760 - i2 / 12))))));
    return r + log(x) - 0.5 / x - series;
}

/* Without a nugget the Matern covariance is linear in sigma^2
 * (Sigma = sigma^2 R(beta, nu)), so dSigma/dsigma^2 = Sigma / sigma^2 and
 *   dl/dsigma^2 = (z^T Sigma^-1 z - N) / (2 sigma^2)
 * exactly, from the quadratic form of the evaluation itself; that component
 * replaces the contraction's (on the INT8-sliced path the quadratic form is
 * good to ~1e-9 while the trace of the sliced inverse is not). */
static void xg_exact_sigma2_grad(const XgField *f, const double *theta, const double *res, double *grad)
{
    if (f->kernel == 0) grad[0] = 0.5 * (res[2] - (double)f->N) / theta[0];
}

/* The gradient's inverse-factor store and contraction partials, each
 * allocated on first use. */
static int xg_grad_workspace(XgField *f)
{
    if (!f->X.d) {
        const int rc = xg_tm_alloc(f->X, f->N, f->C.ts);
        if (rc) return rc;
    }
    const long long blocks = xg_grad_contract_blocks(f->C.ntiles, f->C.ts);
    if (!f->gpart && xg_malloc(&f->gpart, 4 * (size_t)blocks * sizeof(double)) != cudaSuccess) {
        f->gpart = nullptr;
        return xg_fail(XG_ERR_NO_MEMORY, "gradient workspace");
    }
    if (!f->gout && xg_malloc(&f->gout, 4 * sizeof(double)) != cudaSuccess) {
        f->gout = nullptr;
        return xg_fail(XG_ERR_NO_MEMORY, "gradient workspace");
    }
    return XG_OK;
}

/* log-likelihood and its gradient (see gradient_fp64.cu for the steps);
 * grad has 3 entries (4 for the nugget kernel) */
int xg_field_loglik_grad(XgField *f, const double *theta, double *res, double *grad, double *times)
{
    int rc = xg_grad_workspace(f);
    if (rc) return rc;
    if ((rc = xg_check_theta(theta, f->kernel))) return rc;
    const XgMaternParams p = xg_params(theta, f->kernel);
    XgI8Use use(f->C, p); /* the factor's planes serve its inverse */
    rc = xg_field_loglik(f, theta, res, times);
    if (rc) return rc;
    cudaStream_t st = g_xg.stream;
    const double dlogcon = -(log(2.0) + xg_digamma(theta[2]));
    XG_CU(cudaEventRecord(f->ev[0], st));
    xg_solve_transposed(f->C, f->v, f->status, st);
    XgFactorStreams fs;
    fs.st = st;
    fs.st_hi = g_xg.stream_hi;
    fs.ev_panel = f->ev_panel;
    fs.ev_upd = f->ev_upd;
    xg_inverse_product(f->C, f->X, f->status, fs);
    xg_launch_grad_contract(f->C.d, f->C.ij, f->C.ntiles, f->C.nt, f->C.ts, f->x, f->y, f->v, f->N, p, f->kernel,
                            f->metric, dlogcon, f->C.tab, f->gpart, f->gout, st);
    XG_CU(cudaEventRecord(f->ev[3], st));
    double g4[4];
    int sv[2];
    XG_CU(cudaGetLastError());
    XG_CU(cudaMemcpyAsync(g4, f->gout, sizeof g4, cudaMemcpyDeviceToHost, st));
    XG_CU(cudaMemcpyAsync(sv, f->status, sizeof sv, cudaMemcpyDeviceToHost, st));
    XG_CU(cudaStreamSynchronize(st));
    if (sv[0]) {
        f->h_out[3] = sv[0];
        f->h_out[4] = sv[1];
        return xg_read_status(f);
    }
    if (times) {
        float ms = 0;
        cudaEventElapsedTime(&ms, f->ev[0], f->ev[3]);
        times[2] = ms * 1e-3;
    }
    const int np = f->kernel == 1 ? 4 : 3;
    for (int i = 0; i < np; ++i) grad[i] = g4[i];
    /* the contraction kernel accumulates the nugget term in slot 3 */
    xg_exact_sigma2_grad(f, theta, res, grad);
    return XG_OK;
}

/* ------------------------------------------------------------------------- */
/* banded mixed precision                                                    */
/* ------------------------------------------------------------------------- */

static int xg_encode(CUtensorMap *map, CUtensorMapDataType dt, size_t esize, void *base, cuuint64_t cols,
                     cuuint64_t rows, cuuint32_t box_cols, cuuint32_t box_rows,
                     CUtensorMapSwizzle swz = CU_TENSOR_MAP_SWIZZLE_128B)
{
    cuuint64_t dims[2] = {cols, rows};
    cuuint64_t strides[1] = {cols * esize};
    cuuint32_t box[2] = {box_cols, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = g_encode(map, dt, 2, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? XG_OK : xg_fail(XG_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
}

void xg_mixed_destroy(XgMixed *m)
{
    if (!m) return;
    if (m->T.data) cudaFree(m->T.data);
    if (m->T.data32) cudaFree(m->T.data32);
    for (int b = 0; b < 2; ++b) {
        if (m->p64[b]) cudaFree(m->p64[b]);
        if (m->phi[b]) cudaFree(m->phi[b]);
        if (m->plo[b]) cudaFree(m->plo[b]);
    }
    delete m;
}

static int xg_mixed_create(XgMixed **out, int N, int ts, int band, int passes)
{
    *out = nullptr;
    if (ts % 256 != 0) return xg_fail(XG_ERR_BAD_ARGUMENT, "mixed precision needs a tile size multiple of 256 (got %d)", ts);
    if (band < 1) band = 1;
    if (passes != 1 && passes != 3) return xg_fail(XG_ERR_BAD_ARGUMENT, "TF32 passes must be 1 or 3 (got %d)", passes);
    XgMixed *m = new XgMixed();
    const int nt = (N + ts - 1) / ts;
    if (band > nt) band = nt;
    m->band = band;
    m->passes = passes;
    m->T.ts = ts;
    m->T.nt = nt;
    m->T.band = band;
    const size_t tile = (size_t)ts * ts;
    const size_t np = (size_t)nt * ts;
    int rc = XG_OK;
    double *d64 = nullptr;
    float *d32 = nullptr;
    const long long noff = xg_num_offband_tiles(nt, band);
    if (xg_malloc(&d64, (size_t)nt * band * tile * sizeof(double)) != cudaSuccess)
        rc = xg_fail(XG_ERR_NO_MEMORY, "mixed band tiles");
    if (!rc && noff > 0 && xg_malloc(&d32, (size_t)noff * tile * sizeof(float)) != cudaSuccess)
        rc = xg_fail(XG_ERR_NO_MEMORY, "mixed off-band tiles (%.2f GB)", noff * tile * 4.0 / 1e9);
    m->T.data = d64;
    m->T.data32 = d32;
    for (int b = 0; b < 2 && !rc; ++b) {
        if (xg_malloc(&m->p64[b], np * ts * sizeof(double)) != cudaSuccess ||
            xg_malloc(&m->phi[b], np * ts * sizeof(float)) != cudaSuccess ||
            xg_malloc(&m->plo[b], np * ts * sizeof(float)) != cudaSuccess) {
            rc = xg_fail(XG_ERR_NO_MEMORY, "mixed panel buffers");
            break;
        }
        rc = xg_encode(&m->maps[b].p64, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 8, m->p64[b], ts, np, 16, 128);
        if (!rc) rc = xg_encode(&m->maps[b].ahi, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, m->phi[b], ts, np, 32, 128);
        if (!rc) rc = xg_encode(&m->maps[b].bhi, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, m->phi[b], ts, np, 32, 256);
        if (!rc) rc = xg_encode(&m->maps[b].alo, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, m->plo[b], ts, np, 32, 128);
        if (!rc) rc = xg_encode(&m->maps[b].blo, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, m->plo[b], ts, np, 32, 256);
    }
    if (rc) {
        xg_mixed_destroy(m);
        return rc;
    }
    *out = m;
    return XG_OK;
}

/* Mixed factorisation with the z solve fused (v), lookahead as in the FP64
 * path: the panel of step k+1 (POTRF, band TRSM, FP32 TRSM, panel prep) runs
 * on the high-priority stream under the rest of step k's trailing update. */
static void xg_factor_mixed(XgMixed *m, double *v, double *part, int *status, int *info, const XgFactorStreams &fs)
{
    const XgTileArgs &T = m->T;
    const int nt = T.nt;
    const bool la = fs.st_hi != nullptr;
    cudaStream_t sp = la ? fs.st_hi : fs.st;
    /* profiling events, 8 per step: panel start, after POTRF, after TRSM and
     * panel prep, trailing start, after band part 1, after off-band part 1,
     * after band part 2, trailing end */
    cudaEvent_t *pev = fs.pev;
    auto rec = [&](int k, int e, cudaStream_t s) {
        if (pev) cudaEventRecord(pev[8 * k + e], s);
    };
    if (la) cudaEventRecord(fs.ev_upd, fs.st);
    for (int k = 0; k < nt; ++k) {
        const int b = k & 1;
        if (la) cudaStreamWaitEvent(sp, fs.ev_upd, 0);
        rec(k, 0, sp);
        xg_launch_potrf_diag(T, k, v, part, part + nt, v != nullptr, status, info, sp);
        rec(k, 1, sp);
        xg_launch_trsm_panel(T, k, v, v != nullptr, status, sp, k + T.band);
        xg_launch_trsm_panel32(T, k, v, v != nullptr, status, sp);
        if (k + 1 < nt) xg_launch_panel_prep(T, k, m->p64[b], m->phi[b], m->plo[b], m->passes, status, sp);
        rec(k, 2, sp);
        if (la) {
            cudaEventRecord(fs.ev_panel, sp);
            cudaStreamWaitEvent(fs.st, fs.ev_panel, 0);
        }
        rec(k, 3, fs.st);
        if (k + 1 < nt) {
            xg_launch_band_gemm(m->maps[b].p64, T, k, la ? 1 : 0, status, fs.st);
            rec(k, 4, fs.st);
            xg_launch_offband_gemm(m->maps[b], T, k, la ? 1 : 0, m->passes, g_xg.sm_count, status, fs.st);
            rec(k, 5, fs.st);
            if (la) {
                cudaEventRecord(fs.ev_upd, fs.st);
                xg_launch_band_gemm(m->maps[b].p64, T, k, 2, status, fs.st);
                rec(k, 6, fs.st);
                xg_launch_offband_gemm(m->maps[b], T, k, 2, m->passes, g_xg.sm_count - XG_PANEL_SMS, status, fs.st);
            } else {
                rec(k, 6, fs.st);
            }
        } else {
            rec(k, 4, fs.st);
            rec(k, 5, fs.st);
            rec(k, 6, fs.st);
        }
        rec(k, 7, fs.st);
    }
}

/* per-step algorithmic flops of the mixed trailing update: band targets
 * (FP64 DMMA: SYRK ts^2 (ts+1) on the diagonal tile, GEMM 2 ts^3 otherwise)
 * and off-band targets (TF32 tensor cores, 2 ts^3 each) */
static void xg_mixed_step_flops(int nt, int ts, int band, int k, double *band_flops, double *off_flops)
{
    const double t = ts;
    double bf = 0, of = 0;
    for (int j = k + 1; j < nt; ++j) {
        const int rows = nt - j; /* tiles i = j .. nt-1 in column j */
        const int nb = rows < band ? rows : band;
        bf += t * t * (t + 1) + (nb - 1) * 2 * t * t * t;
        if (rows > band) of += (double)(rows - band) * 2 * t * t * t;
    }
    *band_flops = bf;
    *off_flops = of;
}

/* Per-kernel-class times of a banded factorisation (mixed or sliced), from
 * the 8 events per step; launches_per_step counts the panel and trailing
 * launches of one step. */
void xg_field_collect_profile_banded(XgField *f, int band, double launches_per_step)
{
    const int nt = f->C.nt;
    float ms = 0;
    auto el = [&](int a, int b) {
        cudaEventElapsedTime(&ms, f->pev[a], f->pev[b]);
        return ms * 1e-3;
    };
    cudaEventElapsedTime(&ms, f->ev[0], f->ev[1]);
    f->prof[0] += ms * 1e-3;
    for (int k = 0; k < nt; ++k) {
        const int e = 8 * k;
        f->prof[1] += el(e, e + 1);
        f->prof[2] += el(e + 1, e + 2);
        if (k + 1 < nt) {
            f->prof[3] += el(e + 3, e + 7);
            double bfl, ofl;
            xg_mixed_step_flops(nt, f->C.ts, band, k, &bfl, &ofl);
            f->prof[4] += bfl + ofl;
            f->prof[8] += el(e + 4, e + 5) + el(e + 6, e + 7);
            f->prof[9] += ofl;
            f->prof[10] += el(e + 3, e + 4) + el(e + 5, e + 6);
            f->prof[11] += bfl;
        }
    }
    cudaEventElapsedTime(&ms, f->ev[0], f->ev[2]);
    f->prof[7] += ms * 1e-3;
    /* generation and finalize, then per step (upper bound: empty launches are
     * skipped on the host) */
    f->prof[5] += 2 + launches_per_step * nt;
    f->prof[6] += 1;
}

void xg_field_collect_profile_mixed(XgField *f)
{
    /* POTRF, band TRSM, FP32 TRSM, panel prep, two band and two off-band launches */
    xg_field_collect_profile_banded(f, f->mx->band, 8.0);
}

int xg_field_set_mixed(XgField *f, int band, int passes)
{
    if (f->mx && f->mx->band == band && f->mx->passes == passes) return XG_OK;
    if (f->mx) {
        xg_mixed_destroy(f->mx);
        f->mx = nullptr;
    }
    return xg_mixed_create(&f->mx, f->N, f->C.ts, band, passes);
}

int xg_field_loglik_mixed(XgField *f, const double *theta, double *res, double *times)
{
    int rc = xg_check_theta(theta, f->kernel);
    if (rc) return rc;
    if (!f->have_z) return xg_fail(XG_ERR_BAD_ARGUMENT, "no observations: call MLE_zvg or set z first");
    if (!f->mx) {
        rc = xg_field_set_mixed(f, 1, 3);
        if (rc) return rc;
    }
    XgMixed *m = f->mx;
    cudaStream_t st = g_xg.stream;
    const XgMaternParams p = xg_params(theta, f->kernel);
    const size_t Np = (size_t)f->C.nt * f->C.ts;
    XG_CU(cudaMemsetAsync(f->status, 0, 2 * sizeof(int), st));
    XG_CU(cudaMemcpyAsync(f->v, f->z, Np * sizeof(double), cudaMemcpyDeviceToDevice, st));
    XG_CU(cudaEventRecord(f->ev[0], st));
    xg_launch_gen_mixed(m->T, f->C.ij, f->C.ntiles, f->x, f->y, f->N, p, f->metric, st);
    XG_CU(cudaEventRecord(f->ev[1], st));
    XgFactorStreams fs;
    fs.st = st;
    fs.st_hi = g_xg.stream_hi;
    fs.ev_panel = f->ev_panel;
    fs.ev_upd = f->ev_upd;
    fs.pev = f->profiling ? f->pev : nullptr;
    xg_factor_mixed(m, f->v, f->part, f->status, f->info, fs);
    xg_launch_finalize(f->part, f->part + f->C.nt, f->C.nt, f->N, f->out, f->status, f->info, st);
    XG_CU(cudaEventRecord(f->ev[2], st));
    XG_CU(cudaMemcpyAsync(f->h_out, f->out, 5 * sizeof(double), cudaMemcpyDeviceToHost, st));
    XG_CU(cudaGetLastError());
    XG_CU(cudaStreamSynchronize(st));
    if (times) {
        float a = 0, b = 0;
        cudaEventElapsedTime(&a, f->ev[0], f->ev[1]);
        cudaEventElapsedTime(&b, f->ev[1], f->ev[2]);
        times[0] = a * 1e-3;
        times[1] = b * 1e-3;
    }
    if (f->profiling) xg_field_collect_profile_mixed(f);
    rc = xg_read_status(f);
    if (rc) return rc;
    res[0] = f->h_out[0];
    res[1] = f->h_out[1];
    res[2] = f->h_out[2];
    return XG_OK;
}

/* Dense mixed factor L (row-major n x n, zeros above the diagonal) for the
 * parity tests: FP64 band tiles and FP32 off-band tiles widened. */
int xg_mixed_factor_dense(int n, const double *x, const double *y, const double *theta, int kernel, int metric, int ts,
                          int band, int passes, double *out)
{
    XgField *f = nullptr;
    int rc = xg_check_theta(theta, kernel);
    if (rc) return rc;
    rc = xg_field_create(&f, n, ts, x, y, kernel, metric);
    if (rc) return rc;
    rc = xg_field_set_mixed(f, band, passes);
    if (rc) {
        xg_field_destroy(f);
        return rc;
    }
    XgMixed *m = f->mx;
    cudaStream_t st = g_xg.stream;
    cudaMemsetAsync(f->status, 0, 2 * sizeof(int), st);
    xg_launch_gen_mixed(m->T, f->C.ij, f->C.ntiles, f->x, f->y, n, xg_params(theta, kernel), metric, st);
    XgFactorStreams fs;
    fs.st = st;
    fs.st_hi = g_xg.stream_hi;
    fs.ev_panel = f->ev_panel;
    fs.ev_upd = f->ev_upd;
    xg_factor_mixed(m, nullptr, f->part, f->status, f->info, fs);
    cudaError_t e = cudaGetLastError();
    const int nt = m->T.nt, tsz = m->T.ts;
    const size_t tile = (size_t)tsz * tsz;
    std::vector<double> h64((size_t)nt * m->band * tile);
    const long long noff = xg_num_offband_tiles(nt, m->band);
    std::vector<float> h32((size_t)noff * tile);
    int sv[2] = {0, 0};
    if (e == cudaSuccess) e = cudaMemcpyAsync(h64.data(), m->T.data, h64.size() * sizeof(double), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess && noff)
        e = cudaMemcpyAsync(h32.data(), m->T.data32, h32.size() * sizeof(float), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(sv, f->status, sizeof sv, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) rc = xg_cuda_fail(e, "mixed factor");
    if (!rc && sv[0]) rc = xg_fail(sv[0] & XG_ST_NOT_SPD ? XG_ERR_NOT_SPD : XG_ERR_TIMEOUT, "status 0x%x", sv[0]);
    if (!rc)
        for (int r = 0; r < n; ++r)
            for (int c = 0; c < n; ++c) {
                double val = 0.0;
                if (c <= r) {
                    const int i = r / tsz, j = c / tsz;
                    const size_t off = (size_t)(r % tsz) * tsz + (c % tsz);
                    if (i - j < m->band)
                        val = h64[(size_t)xg_slot64(m->T, i, j) * tile + off];
                    else
                        val = h32[(size_t)xg_slot32(i, j, nt, m->band) * tile + off];
                }
                out[(size_t)r * n + c] = val;
            }
    xg_field_destroy(f);
    return rc;
}

/* Copies the lower-tile store of f to a dense row-major n x n array (zeros
 * above the diagonal), after the stream's work; reads the status word. */
static int xg_tiles_to_dense(XgField *f, int n, double *out)
{
    cudaStream_t st = g_xg.stream;
    int rc = XG_OK;
    cudaError_t le = cudaGetLastError();
    if (le != cudaSuccess) return xg_cuda_fail(le, "dense copy launch");
    const int tsz = f->C.ts;
    const size_t tile_elems = (size_t)tsz * tsz;
    double *h = (double *)malloc(f->C.ntiles * tile_elems * sizeof(double));
    if (!h) return xg_fail(XG_ERR_NO_MEMORY, "host copy of the tiles");
    int sv[2] = {0, 0};
    cudaError_t e = cudaMemcpyAsync(h, f->C.d, f->C.ntiles * tile_elems * sizeof(double), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(sv, f->status, sizeof sv, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) rc = xg_cuda_fail(e, "tile download");
    if (!rc && (sv[0] & XG_ST_NOT_SPD)) rc = xg_fail(XG_ERR_NOT_SPD, "not positive definite (pivot %d)", sv[1]);
    if (!rc && sv[0]) rc = xg_fail(XG_ERR_TIMEOUT, "device status word 0x%x", sv[0]);
    if (!rc) {
        for (int r = 0; r < n; ++r)
            for (int c = 0; c < n; ++c) {
                double val = 0.0;
                if (c <= r) {
                    const int i = r / tsz, j = c / tsz;
                    val = h[xg_tile_index(i, j, f->C.nt) * tile_elems + (size_t)(r % tsz) * tsz + (c % tsz)];
                }
                out[(size_t)r * n + c] = val;
            }
    }
    free(h);
    return rc;
}

/* ------------------------------------------------------------------------- */
/* FP64 tiles, INT8-sliced off-band updates                                  */
/* ------------------------------------------------------------------------- */

static void xg_digits_free(XgDigits &D)
{
    if (D.dig) cudaFree(D.dig); /* and scale, behind it */
    D.dig = nullptr;
    D.scale = nullptr;
}

/* digit planes for every tile of M's packed store; the four-digit ones are a
 * workspace that the caller asked for, the seven-digit ones a cache, which
 * takes nobody else's memory */
static int xg_digits_alloc(XgDigits &D, const XgTileMatrix &M, int digits)
{
    const long long rows = M.ntiles * M.ts;
    const size_t plane = (size_t)rows * M.ts;
    if (digits * rows > 0x7fffffffLL)
        return xg_fail(XG_ERR_BAD_ARGUMENT, "N = %d is beyond the sliced path's 2^31-row digit store", M.N);
    D.digits = digits;
    D.plane_rows = (int)rows;
    const XgPart parts[] = {{&D.dig, digits * plane}, {&D.scale, (size_t)rows}};
    if (xg_alloc_parts(parts, 2, digits == 4) != cudaSuccess)
        return xg_fail(XG_ERR_NO_MEMORY, "digit planes (%.2f GB)", digits * (double)plane / 1e9);
    /* both operands are staged in boxes of 128 rows x 64 bytes */
    int rc = xg_encode(&D.map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, D.dig, M.ts, digits * rows, 64, 128,
                       CU_TENSOR_MAP_SWIZZLE_64B);
    if (rc) xg_digits_free(D);
    return rc;
}

void xg_sliced_destroy(XgSliced *s)
{
    if (!s) return;
    xg_digits_free(s->L);
    xg_digits_free(s->X);
    if (s->ev_a) cudaEventDestroy(s->ev_a);
    for (int b = 0; b < 2; ++b)
        if (s->ev_p[b]) cudaEventDestroy(s->ev_p[b]);
    delete s;
}

int xg_sliced_create(XgSliced **out, const XgTileMatrix &M, int digits)
{
    XgSliced *s = new XgSliced();
    int rc = xg_digits_alloc(s->L, M, digits);
    if (!rc && (cudaEventCreateWithFlags(&s->ev_a, cudaEventDisableTiming) != cudaSuccess ||
                cudaEventCreateWithFlags(&s->ev_p[0], cudaEventDisableTiming) != cudaSuccess ||
                cudaEventCreateWithFlags(&s->ev_p[1], cudaEventDisableTiming) != cudaSuccess))
        rc = xg_fail(XG_ERR_CUDA, "sliced lookahead events");
    if (rc) {
        xg_sliced_destroy(s);
        return rc;
    }
    *out = s;
    return XG_OK;
}

/* The matrices that hold seven-digit planes.  Handles may be used from several
 * threads, so the list, i8, i8_users and i8_wanted change under its mutex only;
 * the planes of a matrix in use (XgI8Use) stay until its call ends, which gives
 * them back itself where an allocation waits for them. */
static std::mutex g_i8_mutex;
static std::condition_variable &g_i8_given = *new std::condition_variable(); /* these two outlive handles closed at exit */
static std::vector<XgTileMatrix *> &xg_i8_list()
{
    static std::vector<XgTileMatrix *> *list = new std::vector<XgTileMatrix *>();
    return *list;
}

/* with the mutex held */
static void xg_i8_drop(XgTileMatrix &M)
{
    std::vector<XgTileMatrix *> &list = xg_i8_list();
    list.erase(std::remove(list.begin(), list.end(), &M), list.end());
    xg_sliced_destroy(M.i8);
    M.i8 = nullptr;
    M.i8_factor = false;
}

/* The epilogue weights a product with s_row s_column 254^-6: a subnormal number
 * where the factor (or, for the largest variances, its inverse) is near the low
 * end of the double range.  At sigma^2 = 2^-1000, N = 6700, order 0.5 l was
 * wrong by 1.1e-10 of itself, on DMMA by 9e-15. */
static bool xg_i8_scale_ok(double v) { return v > ldexp(1.0, -800) && v < ldexp(1.0, 800); }

XgI8Use::XgI8Use(XgTileMatrix &m, const XgMaternParams &p) : M(m)
{
    M.i8_scale = xg_i8_scale_ok(p.sigma2 + p.nugget) && (!p.bivariate || xg_i8_scale_ok(p.sigma2b));
    std::lock_guard<std::mutex> lk(g_i8_mutex);
    ++M.i8_users;
}

XgI8Use::~XgI8Use()
{
    std::lock_guard<std::mutex> lk(g_i8_mutex);
    if (--M.i8_users == 0 && M.i8_wanted) {
        if (M.i8) xg_i8_drop(M);
        M.i8_wanted = false;
        g_i8_given.notify_all();
    }
}

static void xg_i8_free(XgTileMatrix &M)
{
    std::lock_guard<std::mutex> lk(g_i8_mutex);
    if (M.i8) xg_i8_drop(M);
    M.i8_factor = M.i8_wanted = false;
    g_i8_given.notify_all();
}

/* Gives the planes of every idle matrix back to the device, or (in_use) waits
 * for those of the matrices in a call; whether there were any */
static bool xg_i8_take_back(bool in_use)
{
    std::unique_lock<std::mutex> lk(g_i8_mutex);
    const std::vector<XgTileMatrix *> held = xg_i8_list();
    for (XgTileMatrix *M : held) {
        if (M->i8_users == 0)
            xg_i8_drop(*M);
        else if (in_use)
            M->i8_wanted = true;
    }
    if (in_use)
        g_i8_given.wait(lk, [] {
            for (XgTileMatrix *M : xg_i8_list())
                if (M->i8_wanted) return false;
            return true;
        });
    return !held.empty();
}

/* Whether the planes of the factor (inverse: of its inverse too) belong to the
 * plan of M: by its size and the device's memory alone, so that the path, and
 * with it the last digits of a result, depend neither on the order of a
 * program's calls nor on what else was allocated when the first was made.  A
 * quarter of what the device has beside the matrix (its planes and the store
 * of the inverse): on 180 GB up to N = 100000, gradients up to 86000. */
static bool xg_i8_planned(const XgTileMatrix &M, bool inverse)
{
    const double e = (double)M.ntiles * M.ts * M.ts;
    return 4.0 * 7.0 * e <= (double)g_xg.memory - (inverse ? 23.0 : 8.0) * e;
}

/* Whether the device has room for them now with three times as much, or a
 * sixteenth of its memory, left for others.  Where it has not, the call runs on
 * DMMA and the next one asks again. */
static bool xg_i8_room(const XgTileMatrix &M)
{
    const size_t bytes = 7 * (size_t)M.ntiles * M.ts * M.ts;
    size_t fr = 0, total = 0;
    return cudaMemGetInfo(&fr, &total) == cudaSuccess && fr >= bytes + std::min(3 * bytes, g_xg.memory / 16);
}

/* The planes of M for a factorisation, allocated where they are wanted and
 * missing; the caller holds an XgI8Use */
static bool xg_i8_acquire(XgTileMatrix &M)
{
    if (M.i8) return true;
    XgSliced *s = nullptr;
    if (!xg_i8_planned(M, false) || !xg_i8_room(M) || xg_sliced_create(&s, M, 7) != XG_OK) return false;
    std::lock_guard<std::mutex> lk(g_i8_mutex);
    M.i8 = s;
    xg_i8_list().push_back(&M);
    return true;
}

static bool xg_i8_acquire_inverse(XgTileMatrix &M)
{
    return M.i8->X.dig || (xg_i8_planned(M, true) && xg_i8_room(M) && xg_digits_alloc(M.i8->X, M, 7) == XG_OK);
}

int xg_field_set_sliced(XgField *f)
{
    if (f->sl) return XG_OK;
    if (f->C.ts % 128 != 0) return xg_fail(XG_ERR_BAD_ARGUMENT, "the sliced path needs a tile size multiple of 128");
    return xg_sliced_create(&f->sl, f->C, 4);
}

/* Factorisation with FP64 tiles and INT8-sliced updates; a column's panel is
 * POTRF and TRSM of the tile column (a window of the tile DAG, with log-det
 * and z solve) and its slicing into digit planes. */
static int xg_factor_sliced(XgTileMatrix &M, XgSliced *sl, double *v, double *part, int *status,
                            const XgFactorStreams &fs)
{
    XgTileArgs T{M.d, M.ts, M.nt};
    const int nt = M.nt, bpt = M.ts / XG_DAG_BLOCK;
    const int nb = (M.N + XG_DAG_BLOCK - 1) / XG_DAG_BLOCK;
    const long long plane = (long long)sl->L.plane_rows * M.ts;
    int *windows = M.dag + xg_dag_words(nb) - nb;
    cudaMemsetAsync(M.dag, 0, sizeof(int) * (size_t)xg_dag_words(nb), fs.st);
    xg_sliced_groups(
        nt, sl, fs,
        [&](int col, int ncol, int k0, int k1, int ctas, cudaStream_t s) {
            if (ncol > 0 && k1 > k0)
                xg_launch_sliced(sl->L, sl->L, T, xg_sl_task(XG_SL_FACTOR, col, ncol, k0, k1), ctas, status, s);
        },
        [&](int c, cudaStream_t s) {
            xg_launch_dag_columns(M, c * bpt, (c + 1) * bpt, windows + c, v, part, status, g_xg.sm_count, s);
            if (fs.pev) cudaEventRecord(fs.pev[8 * c + 2], s);
            if (c + 1 < nt) xg_launch_slice_panel(T, c, 0, sl->L.digits, sl->L.dig, sl->L.scale, plane, status, s);
        });
    return nb;
}

/* Per-kernel-class times of the sliced factorisation from its events:
 * prof[8], prof[9] = seconds and algorithmic flops of the split updates on
 * the main stream (chunks k < j-1 of column j: nearly all the work);
 * prof[10], prof[11] = the same for the last-chunk updates on the panel
 * stream (all chunks of a column without the lookahead). */
static void xg_field_collect_profile_sliced(XgField *f, bool lookahead)
{
    const int nt = f->C.nt;
    const double t = f->C.ts;
    float ms = 0;
    auto el = [&](int a, int b) {
        cudaEventElapsedTime(&ms, f->pev[a], f->pev[b]);
        return ms * 1e-3;
    };
    /* algorithmic flops of `chunks` panel chunks applied to column j */
    auto col_flops = [&](int j, int chunks) {
        return (double)chunks * ((nt - j - 1) * 2.0 * t * t * t + t * t * (t + 1));
    };
    cudaEventElapsedTime(&ms, f->ev[0], f->ev[1]);
    f->prof[0] += ms * 1e-3;
    for (int j = 0; j < nt; ++j) {
        const int e = 8 * j;
        f->prof[1] += el(e + 1, e + 2);
        f->prof[2] += el(e + 2, e + 3);
        const double tb = el(e, e + 1), ta = el(e + 4, e + 5);
        f->prof[3] += ta + tb;
        f->prof[4] += col_flops(j, j);
        if (lookahead) {
            /* on the panel stream: a group's first column by the group before,
             * the others by their own group; U1 of the next group on the main stream */
            const int G = xg_sl_group(nt, f->sl->L.digits), a = j / G * G, b1 = a + 2 * G < nt ? a + 2 * G : nt;
            f->prof[10] += tb;
            f->prof[11] += j > a ? col_flops(j, j - a) : j > 0 ? col_flops(j, G) : 0.0;
            f->prof[8] += ta;
            if (j == a)
                for (int c = a + G; c < b1; ++c) f->prof[9] += col_flops(c, a);
        } else {
            f->prof[8] += tb;
            f->prof[9] += col_flops(j, j);
        }
    }
    cudaEventElapsedTime(&ms, f->ev[0], f->ev[2]);
    f->prof[7] += ms * 1e-3;
    /* generation, finalize; per column two update launches, the panel, slicing */
    f->prof[5] += 2 + 4.0 * nt;
    f->prof[6] += 1;
}

int xg_field_loglik_sliced(XgField *f, const double *theta, double *res, double *times)
{
    int rc = xg_check_theta(theta, f->kernel);
    if (rc) return rc;
    if (!f->have_z) return xg_fail(XG_ERR_BAD_ARGUMENT, "no observations: call MLE_zvg or set z first");
    if (!f->sl) {
        rc = xg_field_set_sliced(f);
        if (rc) return rc;
    }
    cudaStream_t st = g_xg.stream;
    XgTileArgs T{f->C.d, f->C.ts, f->C.nt};
    const XgMaternParams p = xg_params(theta, f->kernel);
    const size_t Np = (size_t)f->C.nt * f->C.ts;
    XG_CU(cudaMemsetAsync(f->status, 0, 2 * sizeof(int), st));
    XG_CU(cudaMemcpyAsync(f->v, f->z, Np * sizeof(double), cudaMemcpyDeviceToDevice, st));
    XG_CU(cudaEventRecord(f->ev[0], st));
    xg_launch_gen(T, f->C.ij, f->C.ntiles, f->x, f->y, f->x, f->y, f->N, f->N, p, f->metric, 1, f->C.tab, st);
    XG_CU(cudaEventRecord(f->ev[1], st));
    XgFactorStreams fs;
    fs.st = st;
    fs.st_hi = g_xg.stream_hi;
    fs.ev_panel = f->ev_panel;
    fs.ev_upd = f->ev_upd;
    fs.pev = f->profiling ? f->pev : nullptr;
    const int np = xg_factor_sliced(f->C, f->sl, f->v, f->part, f->status, fs);
    xg_launch_finalize(f->part, f->part + np, np, f->N, f->out, f->status, f->info, st);
    XG_CU(cudaEventRecord(f->ev[2], st));
    XG_CU(cudaMemcpyAsync(f->h_out, f->out, 5 * sizeof(double), cudaMemcpyDeviceToHost, st));
    XG_CU(cudaGetLastError());
    XG_CU(cudaStreamSynchronize(st));
    if (times) {
        float a = 0, b = 0;
        cudaEventElapsedTime(&a, f->ev[0], f->ev[1]);
        cudaEventElapsedTime(&b, f->ev[1], f->ev[2]);
        times[0] = a * 1e-3;
        times[1] = b * 1e-3;
    }
    if (f->profiling) xg_field_collect_profile_sliced(f, fs.st_hi != nullptr);
    rc = xg_read_status(f);
    if (rc) return rc;
    res[0] = f->h_out[0];
    res[1] = f->h_out[1];
    res[2] = f->h_out[2];
    return XG_OK;
}

/* Dense factor L (row-major n x n, zeros above the diagonal) of the sliced
 * path, for the parity tests. */
int xg_sliced_factor_dense(int n, const double *x, const double *y, const double *theta, int kernel, int metric,
                           int ts, double *out)
{
    XgField *f = nullptr;
    int rc = xg_check_theta(theta, kernel);
    if (rc) return rc;
    rc = xg_field_create(&f, n, ts, x, y, kernel, metric);
    if (!rc) rc = xg_field_set_sliced(f);
    if (rc) {
        xg_field_destroy(f);
        return rc;
    }
    cudaStream_t st = g_xg.stream;
    XgTileArgs T{f->C.d, f->C.ts, f->C.nt};
    cudaMemsetAsync(f->status, 0, 2 * sizeof(int), st);
    xg_launch_gen(T, f->C.ij, f->C.ntiles, f->x, f->y, f->x, f->y, n, n, xg_params(theta, kernel), metric, 1, f->C.tab, st);
    XgFactorStreams fs;
    fs.st = st;
    fs.st_hi = g_xg.stream_hi;
    fs.ev_panel = f->ev_panel;
    fs.ev_upd = f->ev_upd;
    xg_factor_sliced(f->C, f->sl, nullptr, f->part, f->status, fs);
    rc = xg_tiles_to_dense(f, n, out);
    xg_field_destroy(f);
    return rc;
}

/* Gradient with the sliced path: the forward factorisation as
 * xg_field_loglik_sliced, alpha = L^-T v in FP64, the inverse factor
 * X = L^-T by groups of columns (INT8-sliced updates from the digit planes of L
 * and of the already finished columns of X, the FP64 triangular solve with
 * L_bb^T and the slicing of column b of X), S = X X^T by one sliced launch
 * written over the factor, and the FP64 contraction with dSigma/dtheta. */
int xg_field_loglik_grad_sliced(XgField *f, const double *theta, double *res, double *grad, double *times)
{
    int rc = XG_OK;
    if (!f->sl && (rc = xg_field_set_sliced(f))) return rc;
    XgSliced *sl = f->sl;
    if ((rc = xg_grad_workspace(f))) return rc;
    const int ts = f->C.ts, nt = f->C.nt;
    if (!sl->X.dig && (rc = xg_digits_alloc(sl->X, f->C, 4))) return rc;
    rc = xg_field_loglik_sliced(f, theta, res, times);
    if (rc) return rc;
    cudaStream_t st = g_xg.stream;
    const XgMaternParams p = xg_params(theta, f->kernel);
    const double dlogcon = -(log(2.0) + xg_digamma(theta[2]));
    XG_CU(cudaEventRecord(f->ev[0], st));
    xg_solve_transposed(f->C, f->v, f->status, st);
    XgFactorStreams fs;
    fs.st = st;
    fs.st_hi = g_xg.stream_hi;
    fs.ev_panel = f->ev_panel;
    fs.ev_upd = f->ev_upd;
    xg_inverse_product_sliced(f->C, f->X, sl, f->status, fs);
    xg_launch_grad_contract(f->C.d, f->C.ij, f->C.ntiles, nt, ts, f->x, f->y, f->v, f->N, p, f->kernel, f->metric,
                            dlogcon, f->C.tab, f->gpart, f->gout, st);
    XG_CU(cudaEventRecord(f->ev[3], st));
    double g4[4];
    int sv[2];
    XG_CU(cudaGetLastError());
    XG_CU(cudaMemcpyAsync(g4, f->gout, sizeof g4, cudaMemcpyDeviceToHost, st));
    XG_CU(cudaMemcpyAsync(sv, f->status, sizeof sv, cudaMemcpyDeviceToHost, st));
    XG_CU(cudaStreamSynchronize(st));
    if (sv[0]) {
        f->h_out[3] = sv[0];
        f->h_out[4] = sv[1];
        return xg_read_status(f);
    }
    if (times) {
        float ms = 0;
        cudaEventElapsedTime(&ms, f->ev[0], f->ev[3]);
        times[2] = ms * 1e-3;
    }
    const int np = f->kernel == 1 ? 4 : 3;
    for (int i = 0; i < np; ++i) grad[i] = g4[i];
    xg_exact_sigma2_grad(f, theta, res, grad);
    return XG_OK;
}

/* ------------------------------------------------------------------------- */
/* autotuner                                                                 */
/* ------------------------------------------------------------------------- */

/* seconds (CUDA events, generation to result) of one evaluation of f in the
 * given precision after a warm-up one; < 0 on failure; res receives loglik */
static double xg_time_eval(XgField *f, const double *theta, int precision, double *ll)
{
    double res[3], t[3] = {0, 0, 0};
    for (int rep = 0; rep < 2; ++rep) {
        const int rc = precision == 2   ? xg_field_loglik_mixed(f, theta, res, t)
                       : precision == 3 ? xg_field_loglik_sliced(f, theta, res, t)
                                        : xg_field_loglik(f, theta, res, t);
        if (rc) return -1.0;
    }
    if (ll) *ll = res[0];
    return t[0] + t[1];
}

/* Tile size (and, for precision 2, band width) chosen by timing.  Tile
 * sizes 128, 256, 384, 512 (multiples of 256 for precision 2) up to the
 * field size are timed on temporary fields with the same locations and
 * observations; *pf is rebuilt with the fastest.  For precision 2 the band
 * widths 1, 2, 4, 8 are then timed and the fastest whose |dl| / |l| against
 * one FP64 evaluation is <= tol is kept (the most accurate if none is).
 * report receives (ts, seconds) pairs, 4 entries at most. */
int xg_autotune_field(XgField **pf, const double *x, const double *y, const double *theta, int precision, double tol,
                      int *ts_out, int *band_out, double *report)
{
    XgField *f = *pf;
    if (precision == 2 && xg_bivariate(f->kernel))
        return xg_fail(XG_ERR_UNSUPPORTED, "banded mixed precision with bivariate_matern_parsimonious");
    const int N = f->N;
    std::vector<double> z(N);
    int rc = xg_field_get_z(f, z.data(), N);
    if (rc) return rc;
    const int cands[4] = {128, 256, 384, 512};
    int best_ts = f->C.ts, nrep = 0;
    double best_t = -1.0;
    for (int c = 0; c < 4; ++c) {
        const int ts = cands[c];
        if (precision == 2 && ts % 256) continue;
        if (ts > 128 && ts / 2 >= N) continue; /* a single half-empty tile */
        XgField *t = nullptr;
        if (xg_field_create(&t, N, ts, x, y, f->kernel, f->metric)) continue;
        double sec = -1.0;
        if (!xg_field_set_z(t, z.data()) &&
            (precision != 2 || !xg_field_set_mixed(t, f->mx ? f->mx->band : 1, 3)) &&
            (precision != 3 || !xg_field_set_sliced(t)))
            sec = xg_time_eval(t, theta, precision, nullptr);
        xg_field_destroy(t);
        if (sec < 0) continue;
        if (report && nrep < 4) {
            report[2 * nrep] = ts;
            report[2 * nrep + 1] = sec;
            ++nrep;
        }
        if (best_t < 0 || sec < best_t) {
            best_t = sec;
            best_ts = ts;
        }
    }
    if (best_t < 0) return xg_fail(XG_ERR_CUDA, "autotune: no tile size could be timed");
    if (best_ts != f->C.ts) {
        XgField *g = nullptr;
        rc = xg_field_create(&g, N, best_ts, x, y, f->kernel, f->metric);
        if (!rc) rc = xg_field_set_z(g, z.data());
        if (rc) {
            if (g) xg_field_destroy(g);
            return rc;
        }
        g->profiling = false;
        xg_field_destroy(f);
        *pf = f = g;
    }
    *ts_out = best_ts;
    *band_out = 0;
    if (precision == 2) {
        double ll64 = 0;
        if (xg_time_eval(f, theta, 0, &ll64) < 0) return xg_fail(XG_ERR_CUDA, "autotune: FP64 reference evaluation");
        int best_band = 1, acc_band = 1;
        double bt = -1.0, best_err = 1e300;
        const int bands[4] = {1, 2, 4, 8};
        for (int b = 0; b < 4; ++b) {
            if (bands[b] > f->C.nt) break;
            if (xg_field_set_mixed(f, bands[b], 3)) continue;
            double ll = 0;
            const double sec = xg_time_eval(f, theta, 2, &ll);
            if (sec < 0) continue;
            const double err = fabs(ll - ll64) / fabs(ll64);
            if (err <= tol && (bt < 0 || sec < bt)) {
                bt = sec;
                best_band = bands[b];
            }
            if (err < best_err) {
                best_err = err;
                acc_band = bands[b];
            }
        }
        const int band = bt >= 0 ? best_band : acc_band;
        rc = xg_field_set_mixed(f, band, 3);
        if (rc) return rc;
        *band_out = band;
    }
    return XG_OK;
}

int xg_field_get_z(XgField *f, double *z, int n)
{
    if (!f->have_z) return xg_fail(XG_ERR_BAD_ARGUMENT, "no observations generated yet");
    if (n > f->N) n = f->N;
    XG_CU(cudaMemcpy(z, f->z, n * sizeof(double), cudaMemcpyDeviceToHost));
    return XG_OK;
}

/* ------------------------------------------------------------------------- */
/* kriging                                                                   */
/* ------------------------------------------------------------------------- */

void xg_predict_destroy(XgPredict *q)
{
    if (!q) return;
    xg_tm_free(q->C22);
    if (q->xo) cudaFree(q->xo);
    if (q->ev_panel) cudaEventDestroy(q->ev_panel);
    if (q->ev_upd) cudaEventDestroy(q->ev_upd);
    delete q;
}

int xg_predict_create(XgPredict **out, int nmiss, int nobs, int ts)
{
    *out = nullptr;
    int rc = xg_context_require();
    if (rc) return rc;
    if (nmiss <= 0 || nobs <= 0) return xg_fail(XG_ERR_BAD_ARGUMENT, "nZmiss = %d, nZobs = %d", nmiss, nobs);
    XgPredict *q = new XgPredict();
    q->nmiss = nmiss;
    q->nobs = nobs;
    rc = xg_tm_alloc(q->C22, nobs, xg_choose_ts(nobs, ts));
    const size_t Np = (size_t)q->C22.nt * q->C22.ts;
    if (!rc) {
        const size_t nm = (size_t)nmiss;
        const XgPart parts[] = {{&q->xo, Np},   {&q->yo, Np},    {&q->v, Np},
                                {&q->xm, nm},   {&q->ym, nm},    {&q->zact, nm},
                                {&q->zmiss, nm}, {&q->part, 2 * Np / XG_DAG_BLOCK}, {&q->out, 8},
                                {&q->status, 2}};
        cudaError_t e = xg_alloc_parts(parts, 10);
        /* on the stream that fills them: the default stream does not wait for it, nor it for that */
        if (e == cudaSuccess)
            e = cudaMemsetAsync(q->xo, 0, (char *)(q->status + 2) - (char *)q->xo, g_xg.stream);
        if (e != cudaSuccess) rc = xg_fail(XG_ERR_NO_MEMORY, "kriging buffers: %s", cudaGetErrorString(e));
    }
    if (!rc && (cudaEventCreateWithFlags(&q->ev_panel, cudaEventDisableTiming) != cudaSuccess ||
                cudaEventCreateWithFlags(&q->ev_upd, cudaEventDisableTiming) != cudaSuccess))
        rc = xg_fail(XG_ERR_CUDA, "lookahead events");
    if (rc) {
        xg_predict_destroy(q);
        return rc;
    }
    *out = q;
    return XG_OK;
}

int xg_predict_run(XgPredict *q, const double *theta, int kernel, int metric, const double *xm, const double *ym,
                   const double *xo, const double *yo, const double *zobs, const double *zactual, double *zmiss,
                   double *mse, double *mse_parts)
{
    int rc = xg_check_theta(theta, kernel);
    if (rc) return rc;
    if (xg_bivariate(kernel) && ((q->nmiss | q->nobs) & 1))
        return xg_fail(XG_ERR_BAD_ARGUMENT, "bivariate kriging: nZmiss = %d and nZobs = %d must be even (2 x locations)",
                       q->nmiss, q->nobs);
    cudaStream_t st = g_xg.stream;
    const int nmiss = q->nmiss, nobs = q->nobs;
    /* bivariate: nmiss and nobs count matrix rows, two per location */
    const int lmiss = xg_bivariate(kernel) ? nmiss / 2 : nmiss, lobs = xg_bivariate(kernel) ? nobs / 2 : nobs;
    XgTileArgs T{q->C22.d, q->C22.ts, q->C22.nt};
    const XgMaternParams p = xg_params(theta, kernel);
    XgI8Use use(q->C22, p);
    const size_t Np = (size_t)q->C22.nt * q->C22.ts;
    XG_CU(cudaMemsetAsync(q->status, 0, 2 * sizeof(int), st));
    XG_CU(cudaMemsetAsync(q->v, 0, Np * sizeof(double), st));
    XG_CU(cudaMemcpyAsync(q->xo, xo, lobs * sizeof(double), cudaMemcpyHostToDevice, st));
    XG_CU(cudaMemcpyAsync(q->yo, yo, lobs * sizeof(double), cudaMemcpyHostToDevice, st));
    XG_CU(cudaMemcpyAsync(q->v, zobs, nobs * sizeof(double), cudaMemcpyHostToDevice, st));
    XG_CU(cudaMemcpyAsync(q->xm, xm, lmiss * sizeof(double), cudaMemcpyHostToDevice, st));
    XG_CU(cudaMemcpyAsync(q->ym, ym, lmiss * sizeof(double), cudaMemcpyHostToDevice, st));
    if (zactual) XG_CU(cudaMemcpyAsync(q->zact, zactual, nmiss * sizeof(double), cudaMemcpyHostToDevice, st));
    /* C22 = Sigma(obs, obs); POSV: L L^T alpha = zobs */
    xg_launch_gen(T, q->C22.ij, q->C22.ntiles, q->xo, q->yo, q->xo, q->yo, nobs, nobs, p, metric, 1, q->C22.tab, st);
    XgFactorStreams fs;
    fs.st = st;
    fs.st_hi = g_xg.stream_hi;
    fs.ev_panel = q->ev_panel;
    fs.ev_upd = q->ev_upd;
    xg_factor_lookahead(q->C22, q->v, q->part, q->status, q->info(), fs);
    xg_solve_transposed(q->C22, q->v, q->status, st);
    /* zmiss = Sigma(miss, obs) alpha, C12 generated on the fly */
    xg_launch_predict_cross(q->xm, q->ym, nmiss, q->xo, q->yo, nobs, q->v, p, metric, q->zmiss, st);
    if (zactual) xg_launch_mse(q->zact, q->zmiss, nmiss, q->out, st);
    XG_CU(cudaGetLastError());
    int sv[2];
    XG_CU(cudaMemcpyAsync(sv, q->status, sizeof sv, cudaMemcpyDeviceToHost, st));
    XG_CU(cudaMemcpyAsync(zmiss, q->zmiss, nmiss * sizeof(double), cudaMemcpyDeviceToHost, st));
    double m[3] = {-1, -1, -1};
    if (zactual) XG_CU(cudaMemcpyAsync(m, q->out, sizeof m, cudaMemcpyDeviceToHost, st));
    XG_CU(cudaStreamSynchronize(st));
    if (sv[0] & XG_ST_NOT_SPD) return xg_fail(XG_ERR_NOT_SPD, "C22 is not positive definite (pivot %d)", sv[1]);
    if (sv[0]) return xg_fail(XG_ERR_TIMEOUT, "device status word 0x%x", sv[0]);
    *mse = zactual ? m[0] : -1.0;
    if (mse_parts) {
        mse_parts[0] = zactual ? m[1] : -1.0;
        mse_parts[1] = zactual ? m[2] : -1.0;
    }
    return XG_OK;
}

/* ------------------------------------------------------------------------- */
/* dense diagnostics                                                         */
/* ------------------------------------------------------------------------- */

int xg_covariance_dense(int n, const double *x, const double *y, const double *theta, int kernel, int metric, int ts,
                        int factor, double *out)
{
    XgField *f = nullptr;
    int rc = xg_check_theta(theta, kernel);
    if (rc) return rc;
    rc = xg_field_create(&f, n, ts, x, y, kernel, metric);
    if (rc) return rc;
    cudaStream_t st = g_xg.stream;
    XgTileArgs T{f->C.d, f->C.ts, f->C.nt};
    const XgMaternParams p = xg_params(theta, kernel);
    cudaMemsetAsync(f->status, 0, 2 * sizeof(int), st);
    xg_launch_gen(T, f->C.ij, f->C.ntiles, f->x, f->y, f->x, f->y, n, n, p, metric, 1, f->C.tab, st);
    {
        XgI8Use use(f->C, p);
        if (factor) xg_factor(f->C, nullptr, f->part, f->status, f->info, st);
        rc = xg_tiles_to_dense(f, n, out);
    }
    xg_field_destroy(f);
    return rc;
}

int xg_bessel_knu_host(int n, const double *nu, const double *x, double *out)
{
    int rc = xg_context_require();
    if (rc) return rc;
    if (n <= 0) return XG_OK;
    double *d = nullptr;
    XG_CU(xg_malloc(&d, 3 * (size_t)n * sizeof(double)));
    cudaStream_t st = g_xg.stream;
    cudaMemcpyAsync(d, nu, n * sizeof(double), cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(d + n, x, n * sizeof(double), cudaMemcpyHostToDevice, st);
    xg_launch_bessel(d, d + n, n, d + 2 * (size_t)n, st);
    cudaMemcpyAsync(out, d + 2 * (size_t)n, n * sizeof(double), cudaMemcpyDeviceToHost, st);
    cudaError_t e = cudaStreamSynchronize(st);
    cudaFree(d);
    if (e != cudaSuccess) return xg_cuda_fail(e, "bessel");
    return XG_OK;
}

int xg_matern_pairs_host(int n, const double *x1, const double *y1, const double *x2, const double *y2,
                         const double *theta, int kernel, int metric, double *out)
{
    int rc = xg_context_require();
    if (rc) return rc;
    rc = xg_check_theta(theta, kernel);
    if (rc) return rc;
    if (n <= 0) return XG_OK;
    double *d = nullptr;
    XG_CU(xg_malloc(&d, 5 * (size_t)n * sizeof(double)));
    cudaStream_t st = g_xg.stream;
    const double *src[4] = {x1, y1, x2, y2};
    for (int i = 0; i < 4; ++i)
        cudaMemcpyAsync(d + (size_t)i * n, src[i], n * sizeof(double), cudaMemcpyHostToDevice, st);
    xg_launch_matern_pairs(d, d + n, d + 2 * (size_t)n, d + 3 * (size_t)n, n, xg_params(theta, kernel), metric,
                           d + 4 * (size_t)n, st);
    if (cudaGetLastError() != cudaSuccess) {
        cudaFree(d);
        return xg_fail(XG_ERR_CUDA, "matern pairs launch failed");
    }
    cudaMemcpyAsync(out, d + 4 * (size_t)n, n * sizeof(double), cudaMemcpyDeviceToHost, st);
    cudaError_t e = cudaStreamSynchronize(st);
    cudaFree(d);
    if (e != cudaSuccess) return xg_cuda_fail(e, "matern pairs");
    return XG_OK;
}
