/*
 * Piecewise polynomial form of the Matern element for one order.
 *
 * For a fixed order the element is a function of r = d / beta alone, and
 * g(r) = e^r con r^nu K_nu(r) is analytic for r > 0 with its only singularity
 * at r = 0.  On [2^e (1 + m/16), 2^e (1 + (m+1)/16)] that singularity lies at
 * least 33 half-widths from the centre, so interpolation at Chebyshev points
 * converges like (33 + sqrt(33^2 - 1))^-n = 66^-n (Trefethen, Approximation
 * Theory and Approximation Practice, theorem 8.2): nine points leave less than
 * 1e-16 of g for nu <= XG_TAB_NU.  A table of 400 such intervals covers 2^-16 <= r < 2^9; its
 * values come from the direct evaluation (kbessel.cuh), 3600 of them per
 * function, and every element then costs a distance, nine coefficients and
 * one exponential instead of a series or a quadrature with an exponential
 * per node.  Outside the range the direct evaluation is used.
 *
 * The interval and its centre are the leading bits of r, so r minus the
 * centre is exact.  The coefficients are those of the Chebyshev sum about the
 * centre's value, turned into powers of (r - centre): the transform's
 * roundings act on the small differences only.
 */
#ifndef EXAGEOSTAT_B200_MATERN_TAB_CUH
#define EXAGEOSTAT_B200_MATERN_TAB_CUH

#include <math.h>
#include <stdint.h>
#include <string.h>

#include "kbessel.cuh"

#define XG_TAB_NC 9
#define XG_TAB_NINT 400
#define XG_TAB_SIZE (XG_TAB_NINT * XG_TAB_NC)
#define XG_TAB_BASE ((1023 - 16) << 4) /* leading bits of 2^-16 */
#define XG_TAB_NU 5.0

/* Whether tables of functions with the constant c hold them to full precision:
 * the power-8 coefficients are up to 2^168 times the function on the smallest
 * intervals and 2^-80 of it on the largest, so constants near the ends of the
 * double range would overflow or lose bits there. */
XG_HD inline bool xg_tab_scale_ok(double c)
{
    c = fabs(c);
    return c == 0.0 || (c > 1.4996968138956309e-241 && c < 6.668014432879854e+240); /* 2^-800, 2^800 */
}

XG_HD inline uint64_t xg_tab_bits(double r)
{
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(r);
#else
    uint64_t b;
    memcpy(&b, &r, 8);
    return b;
#endif
}
XG_HD inline double xg_tab_double(uint64_t b)
{
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double r;
    memcpy(&r, &b, 8);
    return r;
#endif
}

/* interval of r, or a value >= XG_TAB_NINT (unsigned) outside the table (also for NaN) */
XG_HD inline unsigned xg_tab_index(double r) { return (unsigned)(xg_tab_bits(r) >> 48) - XG_TAB_BASE; }
XG_HD inline double xg_tab_centre(double r)
{
    return xg_tab_double((xg_tab_bits(r) & 0xFFFF000000000000ull) | 0x0000800000000000ull);
}
/* centre and half-width of interval i */
XG_HD inline void xg_tab_interval(int i, double *c, double *hw)
{
    *c = xg_tab_double(((uint64_t)(XG_TAB_BASE + i) << 48) | 0x0000800000000000ull);
    *hw = xg_tab_double((uint64_t)(((XG_TAB_BASE + i) >> 4) - 5) << 52);
}

/* e^r con r^nu K_nu(r) */
XG_HD inline double xg_tab_matern(double r, double nu, double con, const XgTemme &tm)
{
    if (r <= 2.0) return xg_matern_small_c(r, con, tm) * exp(r);
    const double f = con * exp(nu * log(r));
    if (r >= XG_KNU_ASYM_X && nu <= XG_KNU_ASYM_NU) return f * (XG_SQRT_HALF_PI / sqrt(r)) * xg_knu_asym_sum(nu, r);
    return f * xg_knu_scaled_trap(nu, r);
}

/* e^r times dM/dsigma2, dM/dbeta, dM/dnu (xg_matern_grad) */
XG_HD inline void xg_tab_matern_grad(double r, double nu, double con, double sigma2, double beta, double dlogcon,
                                     double *g)
{
    double ek, ekm1, edk;
    if (r >= XG_KNU_ASYM_X && nu <= XG_KNU_ASYM_NU)
        xg_knu_asym3(nu, r, &ek, &ekm1, &edk);
    else
        xg_knu_trap3(nu, r, &ek, &ekm1, &edk);
    const double lr = log(r), f = con * exp(nu * lr), M = f * ek;
    g[0] = M / sigma2;
    g[1] = f * r * ekm1 / beta;
    g[2] = M * (lr + dlogcon) + f * edk;
}

/* the interval's polynomial in powers of r - centre from the values at the
 * nodes t_j = cos((2 j + 1) pi / 18) */
XG_HD inline void xg_tab_coefficients(const double *f, double hw, double *coef)
{
    /* cos(m pi / 18), m = 0 .. 9 */
    const double cs[10] = {1.0,
                           0.98480775301220805937,
                           0.93969262078590838405,
                           0.86602540378443864676,
                           0.76604444311897803520,
                           0.64278760968653932632,
                           0.5,
                           0.34202014332566873304,
                           0.17364817766693034885,
                           0.0};
    const double mid = f[4];
    double a[XG_TAB_NC];
#pragma unroll
    for (int k = 0; k < XG_TAB_NC; ++k) {
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < XG_TAB_NC; ++j) {
            int m = (k * (2 * j + 1)) % 36; /* cos(m pi / 18) */
            if (m > 18) m = 36 - m;
            const double c = m <= 9 ? cs[m] : -cs[18 - m];
            s += (f[j] - mid) * c;
        }
        a[k] = s * ((k == 0 ? 1.0 : 2.0) / XG_TAB_NC);
    }
    const double ih = 1.0 / hw, h2 = ih * ih, h4 = h2 * h2;
    coef[0] = mid + (a[0] - a[2] + a[4] - a[6] + a[8]);
    coef[1] = (a[1] - 3.0 * a[3] + 5.0 * a[5] - 7.0 * a[7]) * ih;
    coef[2] = (2.0 * a[2] - 8.0 * a[4] + 18.0 * a[6] - 32.0 * a[8]) * h2;
    coef[3] = (4.0 * a[3] - 20.0 * a[5] + 56.0 * a[7]) * (h2 * ih);
    coef[4] = (8.0 * a[4] - 48.0 * a[6] + 160.0 * a[8]) * h4;
    coef[5] = (16.0 * a[5] - 112.0 * a[7]) * (h4 * ih);
    coef[6] = (32.0 * a[6] - 256.0 * a[8]) * (h4 * h2);
    coef[7] = 64.0 * a[7] * (h4 * h2 * ih);
    coef[8] = 128.0 * a[8] * (h4 * h4);
}
/* node j of an interval */
XG_HD inline double xg_tab_node(double c, double hw, int j)
{
    const double t[XG_TAB_NC] = {0.98480775301220805937, 0.86602540378443864676,  0.64278760968653932632,
                                 0.34202014332566873304, 0.0,                     -0.34202014332566873304,
                                 -0.64278760968653932632, -0.86602540378443864676, -0.98480775301220805937};
    return c + hw * t[j];
}

/* the polynomial at r (in the table's range); coefficients [interval][9] */
XG_HD inline double xg_tab_poly(const double *tab, unsigned i, double d)
{
    const double *q = tab + i * XG_TAB_NC;
    double s = q[8];
#pragma unroll
    for (int k = 7; k >= 0; --k) s = fma(s, d, q[k]);
    return s;
}

#endif
