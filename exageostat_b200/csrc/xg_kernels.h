/*
 * Internal interface between the host engine and the CUDA kernels.
 */
#ifndef EXAGEOSTAT_B200_KERNELS_H
#define EXAGEOSTAT_B200_KERNELS_H

#include <cuda.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "xg_temme.h"

/* Tile sizes are multiples of 128 up to XG_MAX_TS: the panel TRSM stages
 * 32 x ts doubles in shared memory. */
#define XG_MAX_TS 512

/* A lower-tile matrix on the device (see dense_fp64.cu for the layout).
 * band == 0: every lower tile is FP64 in data, packed (xg_tile_index).
 * band  > 0: banded mixed precision -- data holds only the FP64 band tiles
 * (0 <= i - j < band, compact: slot j * band + (i - j)), data32 the FP32
 * off-band tiles (compact, xg_slot32). */
struct XgTileArgs {
    double *data;
    int ts; /* tile size */
    int nt; /* tiles per side */
    int band = 0;
    float *data32 = nullptr;
    long long tile_off = 0; /* first tile of this matrix inside a shared TMA tensor (batches) */
    /* band == 0 only: restricts the DMMA trailing update to the targets
     * 0 <= i - j < band_targets (the others go to the INT8-sliced kernel) */
    int band_targets = 0;
    /* optional: ts x 32 doubles receiving the inverses of the 32 x 32
     * diagonal blocks of the current panel's L_kk (written by
     * xg_launch_potrf_tiled); with it the panel TRSM applies them as DMMA
     * products instead of a serial substitution */
    double *dinv = nullptr;
};

__host__ __device__ inline long long xg_slot64(const XgTileArgs &T, int i, int j)
{
    if (T.band) return (long long)j * T.band + (i - j);
    return (long long)j * T.nt - (long long)j * (j - 1) / 2 + (i - j);
}

/* off-band tile (i, j), i - j >= band: column j holds nt - j - band tiles */
__host__ __device__ inline long long xg_slot32(int i, int j, int nt, int band)
{
    const long long M = nt - band;
    return (long long)j * M - (long long)j * (j - 1) / 2 + (i - j - band);
}

__host__ __device__ inline long long xg_num_offband_tiles(int nt, int band)
{
    const long long M = nt - band;
    return M > 0 ? M * (M + 1) / 2 : 0;
}

/* Matern parameters of one covariance evaluation.  con = sigma^2 /
 * (2^(nu-1) Gamma(nu)) is computed on the host exactly as core_zcmg.c:976-978;
 * half_integer = 0, 1, 2 selects the closed form for nu = 0.5, 1.5, 2.5
 * (exact match of nu), -1 the general Bessel path. */
struct XgMaternParams {
    double sigma2;
    double beta;
    double nu;
    double nugget; /* tau^2, added on the zero-distance branch only */
    double con;
    int half_integer;
    /* bivariate parsimonious Matern (kernel 2): rows and columns interleave
     * the two variables of each location (index 2 l + v); sigma2, nu, con
     * above are variable 0's, these variable 1's and the cross block's
     * (core_zcmg.c:1628-1651) */
    int bivariate;
    double sigma2b, nu2, con2, nu12, con12, cross0;
    /* scales of variable 1 and of the cross covariance (beta is variable 0's):
     * all three equal beta for the parsimonious kernel; the flexible kernel
     * (kernel 3, core_zcmg.c:1514-1580) has one per component */
    double beta2, beta12;
    /* Temme's order constants of nu (univariate kernels, general nu) */
    XgTemme tm;
};

/* One field of a batch of independent fields sharing one tile store. */
struct XgBField {
    long long tile_off; /* first packed tile of the field in the batch store */
    long long vec_off;  /* first entry of its vectors (x, y, z, v); a multiple of ts */
    long long part_off; /* first entry of its partial sums (2 nb) */
    int N, nt, nb;      /* nb: 128-blocks per side */
    int kernel;
    XgMaternParams p;   /* this evaluation's parameters */
};

/* task types of the right-looking plan (exageostat_b200_batch_plan) */
#define XG_TASK_POTRF 0
#define XG_TASK_TRSM 1
#define XG_TASK_GEMM 2

/* The fields taking part in one batched launch and the CTA ranges they own. */
struct XgBStep {
    const int *fields;          /* nact field indices */
    const long long *blk_start; /* nact + 1 prefix sums of CTAs */
    int nact;
};

/* field owning CTA `bid` of a batched launch, and the CTA index within it */
__device__ inline int xg_batch_resolve(const XgBStep &S, long long bid, long long *local)
{
    int lo = 0, hi = S.nact - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (S.blk_start[mid] <= bid)
            lo = mid;
        else
            hi = mid - 1;
    }
    *local = bid - S.blk_start[lo];
    return S.fields[lo];
}

/* (i, j) of packed lower tile t of an nt x nt tile grid */
__device__ inline int2 xg_tile_decode_fast(long long t, int nt)
{
    /* column j starts at j nt - j (j - 1) / 2 */
    const double h = nt + 0.5;
    int j = (int)(h - sqrt(h * h - 2.0 * (double)t));
    if (j < 0) j = 0;
    while (j > 0 && (long long)j * nt - (long long)j * (j - 1) / 2 > t) --j;
    while ((long long)(j + 1) * nt - (long long)(j + 1) * j / 2 <= t) ++j;
    return make_int2(j + (int)(t - ((long long)j * nt - (long long)j * (j - 1) / 2)), j);
}

/* tile_dag.cu: the whole Cholesky of one or more fields in one persistent
 * launch, a dataflow of 128 x 128 blocks. */
#define XG_DAG_BLOCK 128
/* device words of a field's DAG state: next task, abort flag, block flags, then
 * a next-task word per window of columns */
static inline long long xg_dag_words(int nb) { return 2 + (long long)nb * (nb + 1) / 2 + nb; }
/* the same of its backward solve: next task, abort flag, a flag per block */
static inline long long xg_trsv_words(int nb) { return 2 + (long long)nb; }
struct XgDagField {
    long long tile_off; /* first packed tile inside the tile store */
    long long vec_off;  /* first entry of v */
    long long part_off; /* partial sums: nb log-det, nb |v_J|^2 */
    long long flag_off; /* nb (nb + 1) / 2 block flags */
    long long tflag_off; /* nb flags of the backward solve */
    long long dinv_off; /* first row of the inverted 32 x 32 diagonal blocks (32 doubles a row) */
    int nt, nb;         /* tiles per side; 128-blocks per side that hold rows < N */
};
struct XgDag {
    double *data; /* the tile store behind the TMA map */
    int ts;
    XgDagField one;       /* a single field (tasks == nullptr: ntasks blocks in block-column order) */
    int J0;               /* first block column; the columns before it are applied already */
    const XgDagField *F;  /* several fields */
    const int4 *tasks;    /* (field, I, J, -) in an order that never puts a block before its operands */
    long long ntasks;
    unsigned *next;       /* zero on launch: tasks taken so far */
    int *abort;           /* zero on launch; set by a wait that timed out */
    int *flags;           /* zero on launch */
    double *dinv, *v, *part; /* v may be null */
    int *status;          /* two words per field: status, info */
};
cudaError_t xg_dag_kernels_configure();

/* rows_dag.cu: row blocks solved against the factor, one persistent launch */
#define XG_ROWS_INVERSE 0
#define XG_ROWS_RHS 1
#define XG_ROWS_MAX_SYS 3
struct XgRowsField {
    long long l_off, y_off; /* first packed tile of the factor and of the rows */
    long long flag_off;     /* INVERSE: nb (nb + 1) / 2 flags; RHS: nb mr */
    long long dinv_off;     /* first row of the inverted 32 x 32 diagonal blocks */
    int nt, nb;             /* tiles and 128-blocks per side of the factor */
    int mt, mr;             /* RHS: tile rows, 128-row blocks that are not padding */
};
struct XgRowsMaps {
    CUtensorMap y[XG_ROWS_MAX_SYS], l[XG_ROWS_MAX_SYS];
};
struct XgRows {
    double *y[XG_ROWS_MAX_SYS];          /* rows (solved in place, INVERSE: written) */
    const double *dinv[XG_ROWS_MAX_SYS];
    double *s;                           /* INVERSE: the factor's store, receives S */
    int ts, nsys, J0;                    /* J0: first block column of a window (INVERSE, no products) */
    int lower;                           /* RHS: as many rows as columns, only the blocks I >= J */
    XgRowsField one;
    const XgRowsField *F;
    const int4 *tasks;                   /* (field, I, J, product?); null: a single field, every task */
    long long ntasks;
    unsigned *next;                      /* zero on launch, as abort and flags */
    int *abort, *flags;
    long long sys_flags;                 /* flags per system */
    int *status;
};
cudaError_t xg_rows_kernels_configure();
void xg_launch_rows(int mode, const XgRowsMaps &M, const XgRows &G, int max_ctas, cudaStream_t st);

void xg_launch_dag(const CUtensorMap &map, const XgDag &G, int max_ctas, cudaStream_t st);

cudaError_t xg_kernels_configure();
size_t xg_potrf_smem_bytes(int ts);
size_t xg_trsm_smem_bytes(int ts);
size_t xg_gemm_smem_bytes();

/* covariance tiles; tab: xg_tab_doubles() doubles of workspace for the
 * piecewise polynomial form, or null for the direct evaluation */
void xg_launch_gen(const XgTileArgs &T, const int2 *tile_ij, long long ntiles, const double *xr, const double *yr,
                   const double *xc, const double *yc, int n_rows, int n_cols, const XgMaternParams &p, int metric,
                   int identity_pad, double *tab, cudaStream_t st);
void xg_launch_potrf_diag(const XgTileArgs &T, int k, double *v, double *part_logdet, double *part_dot, int with_rhs,
                          int *status, int *info, cudaStream_t st);
void xg_launch_trsm_panel(const XgTileArgs &T, int k, double *v, int with_rhs, const int *status, cudaStream_t st,
                          int i1 = -1);
/* POTRF(k, k) with the fused log-det and solve, by 128 x 128 sub-blocks on
 * several CTAs (map: the TMA view of the tile store); fills T.dinv too */
void xg_launch_potrf_tiled(const CUtensorMap &map, const XgTileArgs &T, int k, double *v, double *part_logdet,
                           double *part_dot, int with_rhs, int *status, int *info, cudaStream_t st);
int xg_potrf_tiled_launches(int ts);
void xg_launch_syrk_gemm(const CUtensorMap &map, const XgTileArgs &T, int k, int *status, cudaStream_t st,
                         int part = 0);

/* matern_tab.cu: tiles of general order from piecewise polynomial tables.
 * Smallest field that builds them: the build takes 9 us, one direct element's
 * own latency as much; an evaluation of 256 locations takes 135 us with the
 * table and 172 us without, one of 1024 455 and 514 us. */
#define XG_TAB_MIN_N 64
cudaError_t xg_tab_kernels_configure(int sm_count);
size_t xg_tab_doubles();
/* whether the tables cover the orders of p and pay for n locations */
bool xg_tab_covers(const XgMaternParams &p, int n);
void xg_launch_gen_tab(const XgTileArgs &T, const int2 *tile_ij, long long ntiles, const double *xr, const double *yr,
                       const double *xc, const double *yc, int n_rows, int n_cols, const XgMaternParams &p, int metric,
                       int identity_pad, double *tab, cudaStream_t st);
/* the three derivative tables of p into tab, then what reads them */
void xg_launch_grad_tables(const XgMaternParams &p, double dlogcon, double *tab, cudaStream_t st);
long long xg_grad_contract_tab_blocks(long long ntiles, int ts);
void xg_launch_grad_contract_tab(const double *S, long long ntiles, int nt, int ts, const double *x, const double *y,
                                 const double *alpha, int N, const XgMaternParams &p, int kernel, int metric,
                                 double dlogcon, const double *tab, double *part, cudaStream_t st);
void xg_launch_dsigma_full_tab(double *D, int nt, int ts, const double *x, const double *y, int N,
                               const XgMaternParams &p, double dlogcon, int metric, int which, const double *tab,
                               cudaStream_t st);

/* mixed.cu: banded mixed precision */
struct XgMixedMaps {
    CUtensorMap p64;           /* FP64 panel copy, boxes 128 x 16 (DMMA band targets) */
    CUtensorMap ahi, bhi;      /* TF32 "hi" panel, boxes 128 x 32 and 256 x 32 (FP32) */
    CUtensorMap alo, blo;      /* TF32 "lo" panel */
};
cudaError_t xg_mixed_kernels_configure();
void xg_launch_gen_mixed(const XgTileArgs &T, const int2 *tile_ij, long long ntiles, const double *x, const double *y,
                         int n, const XgMaternParams &p, int metric, cudaStream_t st);
/* panel TRSM of column k by 128-column blocks (TMA-fed DMMA GEMMs and in-block
 * solves with the inverted 32 x 32 diagonal blocks in T.dinv); ts a multiple of 128 */
void xg_launch_trsm_gemm(const CUtensorMap &map, const XgTileArgs &T, int k, double *v, int with_rhs, int *status,
                         cudaStream_t st);
void xg_launch_trsm_panel32(const XgTileArgs &T, int k, double *v, int with_rhs, const int *status, cudaStream_t st);
void xg_launch_panel_prep(const XgTileArgs &T, int k, double *p64, float *phi, float *plo, int passes,
                          const int *status, cudaStream_t st);
void xg_launch_band_gemm(const CUtensorMap &p64map, const XgTileArgs &T, int k, int part, int *status,
                         cudaStream_t st);
void xg_launch_offband_gemm(const XgMixedMaps &maps, const XgTileArgs &T, int k, int part, int passes, int sm_count,
                            int *status, cudaStream_t st);
/* sliced.cu: FP64 tiles, trailing updates on INT8 tensor cores (four digit slices), left-looking.
 * One launch of xg_sliced_left_kernel computes, for each output tile, C (+)= sign sum_k A_k B_k^T
 * over panel chunks k, with A_k, B_k read from digit stores:
 *   XG_SL_FACTOR : ncol columns of the Cholesky factor from col on, chunks k0 <= k < k1:
 *                  L(i,j) -= sum L(i,k) L(j,k)^T
 *   XG_SL_INVERSE: ncol columns of X = L^-T from col on (X(a,b) at slot (b,a)), chunks k0 <= c < k1:
 *                  X(a,b) -= sum_{a<=c} X(a,c) L(b,c)^T, a < k1; the window that holds chunk a is
 *                  X(a,b)'s first and overwrites it
 *   XG_SL_SYRK   : S = X X^T into the lower tiles: S(a,b) = sum_{c>=a} X(a,c) X(b,c)^T */
#define XG_SL_FACTOR 0
#define XG_SL_INVERSE 1
#define XG_SL_SYRK 2
struct XgSlTask {
    int mode;
    int col, ncol; /* target columns (factor, inverse) */
    int k0, k1;    /* chunk window */
    double sign;   /* -1: C -= sum; +1: C += sum */
};
cudaError_t xg_sliced_kernels_configure();
/* a digit store: `digits` planes of plane_rows rows (ts bytes each), one scale per row */
struct XgDigits {
    int digits = 4, plane_rows = 0;
    int8_t *dig = nullptr;
    double *scale = nullptr;
    CUtensorMap map; /* boxes of 128 rows x 64 bytes, 64-byte swizzle */
};
void xg_launch_slice_panel(const XgTileArgs &T, int k, int row_mode, int digits, int8_t *dig, double *scale,
                           long long plane, const int *status, cudaStream_t st);
void xg_launch_sliced(const XgDigits &A, const XgDigits &B, const XgTileArgs &T, const XgSlTask &S, int max_ctas,
                      int *status, cudaStream_t st);

void xg_launch_finalize(const double *part_logdet, const double *part_dot, int nt, int N, double *out,
                        const int *status, const int *info, cudaStream_t st);

/* batched fields (every field's strips in one launch) */
void xg_launch_batch_gen(const XgTileArgs &base, const XgBField *F, int nfields, const XgBStep &S, long long blocks,
                         const double *x, const double *y, int metric, double *tab, cudaStream_t st);
void xg_launch_batch_finalize(const XgBField *F, int nfields, const double *part, double *out, cudaStream_t st);
/* solve.cu */
void xg_launch_trmv_lower(const XgTileArgs &T, const double *e, double *z, const int *status, cudaStream_t st);
/* v <- L^-T v in one launch, with the inverted 32 x 32 diagonal blocks that
 * the factorisation kept */
struct XgTrsv {
    const double *data;
    int ts;
    XgDagField one;      /* a single field (tasks == nullptr) */
    const XgDagField *F; /* several */
    const int2 *tasks;   /* (field, J), every field's columns in descending order */
    long long ntasks;
    unsigned *next;      /* zero on launch */
    int *abort, *flags;  /* zero on launch */
    const double *dinv;
    double *v;
    int *status;
};
cudaError_t xg_solve_kernels_configure();
void xg_launch_trsv_lower_t(const XgTrsv &G, int max_ctas, cudaStream_t st);
void xg_launch_predict_cross(const double *xm, const double *ym, int nmiss, const double *xo, const double *yo,
                             int nobs, const double *alpha, const XgMaternParams &p, int metric, double *zmiss,
                             cudaStream_t st);
void xg_launch_mse(const double *zactual, const double *zmiss, int nmiss, double *out, cudaStream_t st);
void xg_launch_matern_pairs(const double *x1, const double *y1, const double *x2, const double *y2, int n,
                            const XgMaternParams &p, int metric, double *out, cudaStream_t st);

void xg_launch_bessel(const double *nu, const double *x, int n, double *out, cudaStream_t st);

/* gradient_fp64.cu */
cudaError_t xg_gradient_kernels_configure();
/* zeros the diagonal tiles of a lower-tile store */
void xg_launch_zero_diag(double *X, int nt, int ts, cudaStream_t st);
void xg_launch_rhs_tri_product(const CUtensorMap &mapA, const CUtensorMap &mapB, double *C, int mt, int nt, int ts,
                               int *status, cudaStream_t st);
long long xg_grad_contract_blocks(long long ntiles, int ts);
void xg_launch_grad_contract(const double *S, const int2 *tile_ij, long long ntiles, int nt, int ts, const double *x,
                             const double *y, const double *alpha, int N, const XgMaternParams &mp, int kernel,
                             int metric, double dlogcon, double *tab, double *part, double *out, cudaStream_t st);

/* assess.cu (Fisher information, MLOE / MMOM) */
void xg_launch_cross_gen_r(double *D, int mt, int nt, int ts, const double *xm, const double *ym, int nmiss,
                           const double *xo, const double *yo, int nobs, const XgMaternParams &p, int metric,
                           cudaStream_t st);
void xg_launch_reverse_factor(double *L, const int2 *ij, double *dinv, int nt, int ts, int used, cudaStream_t st);
void xg_launch_reverse_columns(double *dst, const double *src, int mt, int nt, int ts, cudaStream_t st);
void xg_launch_tile_transpose(double *D, long long ntiles, int ts, cudaStream_t st);
void xg_launch_mloe_terms(const double *A, const double *U, const double *T, const double *V, int mt, int nt, int ts,
                          int nmiss, double sigma2_t, double sigma2_a, double *terms, cudaStream_t st);
void xg_launch_lower_transpose(double *Y, int nsys, int nt, int ts, cudaStream_t st);
void xg_launch_dsigma_full(double *D, int nt, int ts, const double *x, const double *y, int N,
                           const XgMaternParams &p, double dlogcon, int metric, int which, double *tab,
                           cudaStream_t st);
void xg_launch_fisher_trace(const double *W, int np, int nt, int ts, int N, double sigma2, double nugget, double *part,
                            int nctas, cudaStream_t st);

#endif
