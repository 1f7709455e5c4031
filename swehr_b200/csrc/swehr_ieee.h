/*
 * swehr_ieee.h -- IEEE-754 quotients and square roots of doubles without a
 * branch, for operands of middling size, shared by the CUDA kernels and the
 * CPU tests.
 *
 * A wet FP64 cell has about a hundred quotients and roots; written out as plain
 * multiply-adds the independent ones overlap.  What they are not exact for is a
 * value that the caller collects over a whole cell (FastF64 in swehr_tile.cuh),
 * and a cell with such an operand is computed again with plain operators.
 * Measured on the 4096^2 domain in ponded flow (7 classes, B200): FP64
 * update 6.29 ms with the operators, 4.24 ms with these; a step on the 3 x 51
 * example 34 and 26 us.
 *
 * Method.  A reciprocal estimate y of 1/b with residual e = 1 - b y is refined by
 * y (1 + e + e^2), an estimate y of x^(-1/2) with e = 1 - x y^2 by
 * y (1 + e/2 + 3 e^2/8): the third-order iterations of the family of A. S.
 * Householder ("The Numerical Treatment of a Single Nonlinear Equation", 1970),
 * the binomial series of 1/(1 - e) and (1 - e)^(-1/2) cut after the square.  The
 * quotient is q = a y corrected by the exact remainder r = a - b q (P. W.
 * Markstein, "Computation of elementary functions on the IBM RISC System/6000
 * processor", IBM J. Res. Dev. 34, 1990).  Why the result is the rounded quotient, for
 * 1 <= b < 2 and y the double next to 1/b, i.e. within 2^-54 of it (a scaling
 * by powers of two changes nothing while no step leaves the normal range):
 *   - away from the midpoint of two neighbouring doubles q + r y rounds
 *     correctly, its error before rounding is below 2^-52 ulp;
 *   - a quotient is never a midpoint, and its distance to one is at least
 *     2^-54 ulp (2/b).  Near a midpoint m the product a y lies within one ulp
 *     of m, so q is m +- ulp/2, r is exact, and q + r y misses a/b by at most
 *     ulp/2 * 2^-54 b, less than that distance as b < 2.
 * The reciprocal's last step carries the square of its residual, rounded up:
 * without it the reciprocal of a significand of ones, which lies 2^-107 above
 * a midpoint, would be the double below.
 * The square root is x y corrected once by its exact remainder x - g^2 with
 * y ~ 1/sqrt(x); the arguments whose root lies near a midpoint satisfy
 * k^2 = -c (mod 2^54) for a small c, a handful for each c, and the tests run
 * them all for |c| < 2000.
 */
#ifndef SWEHR_IEEE_H
#define SWEHR_IEEE_H

#include "swehr_math.h"

/* a - b q rounded down: exact wherever it matters, and -0 where it is zero,
 * so that the correction keeps the sign of a zero quotient */
SW_HD double sw_remainder(double b, double q, double a)
{
#ifdef __CUDACC__
    return __fma_rd(-b, q, a);
#else
    const double r = fma(-b, q, a);
    return r == 0 ? -0.0 : r;
#endif
}

/* e + e^2 rounded up */
SW_HD double sw_square_up(double e)
{
#ifdef __CUDACC__
    return __fma_ru(e, e, e);
#else
    const double u = fma(e, e, e);
    return fma(e, e, -(u - e)) > 0 ? nextafter(u, INFINITY) : u;
#endif
}

/* 1/b from an estimate y within 2^-18 of it, relatively: a cubic step (error
 * below 2^-54), then another */
SW_HD double sw_rcp_refine(double b, double y)
{
    double e = fma(-b, y, 1.0);
    const double u = fma(e, e, e);
    y = fma(y, u, y);
    e = fma(-b, y, 1.0);
    return fma(y, sw_square_up(e), y);
}

/* a / b, b > 0, with y = sw_rcp_refine(b, ..); both of middling size or a zero */
SW_HD double sw_quot(double a, double b, double y)
{
    const double q = a * y;
    const double r = sw_remainder(b, q, a);
    return fma(r, y, q);
}

/* the same for any dividend below 2^501, a subnormal result included, and b in
 * [2^-200, 2^52): the quotient of a 2^400, which lies in the normal range, is scaled
 * back, which rounds a second time where the result is subnormal (last place
 * 2^-1074, 2^-674 scaled).  The remainder there, a multiple of ulp(b) 2^-674
 * below b 2^-674, is exact and says whether the nearest place is the next one; a
 * tie is one of the first quotient too, rounded to even by the scaling. */
SW_HD double sw_quot_tiny(double a, double b, double y)
{
    const double s = a * 0x1p400;
    double q = sw_quot(s, b, y) * 0x1p-400;
    const double r = fma(-b, q * 0x1p400, s);
    if (fabs(q) < 0x1p-1022 && fabs(r) > b * 0x1p-675) q += copysign(0x1p-1074, r);
    return q;
}

/* sqrt(x) from an estimate y within 2^-18 of 1/sqrt(x), relatively; x > 0 of
 * middling size */
SW_HD double sw_sqrt_refine(double x, double y)
{
    double g = x * y;
    const double e = fma(-g, y, 1.0);
    const double p = fma(e, 0.375, 0.5);
    y = fma(y * e, p, y);                     /* error 5/16 e^3 */
    g = x * y;
    const double d = fma(-g, g, x);
    return fma(d, 0.5 * y, g);
}

#ifdef __CUDACC__
SW_HD double sw_rcp(double b)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    return sw_rcp_refine(b, y);
}

/* sqrt(x), x > 0 */
SW_HD double sw_sqrt_pos(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return sw_sqrt_refine(x, y);
}

/* sqrt(x), or +0 for a zero of either sign (pow(x, 0.5)) */
SW_HD double sw_sqrt_mid(double x)
{
    const double g = sw_sqrt_pos(x);
    return ((__double2hiint(x) & 0x7fffffff) | __double2loint(x)) == 0 ? 0.0 : g;
}

/* Sizes, tested on the high word read as a float: its order is that of the
 * double, a NaN or an infinity compares as too large or not at all, and
 * tests of one value chain into one predicate (joined by & and |: a
 * short-circuit would be a branch).  "Middling" is
 * [2^-300, 2^301): quotients of such operands, their remainders and the
 * quotients of those quotients stay inside the normal range. */
#define SW_MID_LO 0x2D300000
#define SW_MID_HI 0x52C00000
SW_HD float sw_hi_float(double x) { return __int_as_float(__double2hiint(x)); }
SW_HD bool sw_below(double x, int hi) { return fabsf(sw_hi_float(x)) < __int_as_float(hi); }
SW_HD bool sw_small(double x) { return sw_below(x, SW_MID_HI); }
SW_HD bool sw_zero(double x) { return ((__double2hiint(x) & 0x7fffffff) | __double2loint(x)) == 0; }
SW_HD bool sw_mid_pos(double x)
{
    const float f = sw_hi_float(x);
    return (f >= __int_as_float(SW_MID_LO)) & (f < __int_as_float(SW_MID_HI));
}
SW_HD bool sw_mid_or_zero(double x)
{
    return ((fabsf(sw_hi_float(x)) >= __int_as_float(SW_MID_LO)) | sw_zero(x)) & sw_small(x);
}

/* A dividend may be as small as 2^-860 over a divisor below 2^52: the quotient
 * is above 2^-913, its remainder a multiple of 2^-965, and the same holds once
 * more for that quotient over a constant below 2^50.  What suspended mass
 * settles to after the rain lies below that too (sw_tiny), down to the smallest
 * subnormals, where a decay by less than a half rounds to no decay at all. */
#define SW_LOW 0x0A300000
#define SW_DEPTH_LO 0x33700000
#define SW_DEPTH_HI 0x43300000
SW_HD bool sw_tiny(double x) { return sw_below(x, SW_LOW) & !sw_zero(x); }
SW_HD bool sw_low_or_zero(double x)
{
    return ((fabsf(sw_hi_float(x)) >= __int_as_float(SW_LOW)) | sw_zero(x)) & sw_small(x);
}
/* a divisor in [2^-200, 2^52) */
SW_HD bool sw_mid_depth(double x)
{
    const float f = sw_hi_float(x);
    return (f >= __int_as_float(SW_DEPTH_LO)) & (f < __int_as_float(SW_DEPTH_HI));
}

/* The polynomials' coefficients in the constant bank: a multiply-add takes its
 * operand from there, while an immediate double is moved into a register pair
 * at every use (4096^2, ponded flow: FP64 update -0.7 %). */
enum { K_INVLN2N, K_LN2N_HI, K_LN2N_LO, K_INVFACT6, K_INVFACT5, K_INVFACT4, K_INVFACT3, K_ATANH_C11, K_ATANH_C9, K_ATANH_C7, K_ATANH_C5, K_ATANH_C3, K_LN2_HI, K_LN2_LO, K_COUNT };
static __device__ __constant__ double sw_kc[K_COUNT] = {
    SW_INVLN2N, SW_LN2N_HI, SW_LN2N_LO, SW_INVFACT6, SW_INVFACT5,
    SW_INVFACT4, SW_INVFACT3, SW_ATANH_C11, SW_ATANH_C9, SW_ATANH_C7,
    SW_ATANH_C5, SW_ATANH_C3, SW_LN2_HI, SW_LN2_LO};

/* sw_exp_core for |x| <= 700: the same operations, the integer taken from
 * the shifted sum's low word and the scale added to the high word */
SW_HD double sw_exp_mid(double x, double xlo)
{
    const double t = fma(x, sw_kc[K_INVLN2N], SW_SHIFT);
    const double kd = t - SW_SHIFT;
    const int k = __double2loint(t), j = k & 63, m = k >> 6;
    double r = fma(-kd, sw_kc[K_LN2N_HI], x);
    r = fma(-kd, sw_kc[K_LN2N_LO], r);
    r = r + xlo;
    double q = fma(r, sw_kc[K_INVFACT6], sw_kc[K_INVFACT5]);
    q = fma(r, q, sw_kc[K_INVFACT4]);
    q = fma(r, q, sw_kc[K_INVFACT3]);
    q = fma(r, q, SW_INVFACT2);
    const double r2 = r * r;
    const double p = fma(r2, q, r);
    const double th = sw_exp2_hi[j];
    const double y = th + fma(th, p, sw_exp2_lo[j]);
    return __hiloint2double(__double2hiint(y) + (m << 20), __double2loint(y));
}

/* |x| <= 700 (false for a NaN) */
SW_HD bool sw_exp_fits(double x) { return sw_below(x, 0x4085E000); }

/* x below -746 (by 2^-10 or more: the high word decides), where exp rounds to
 * zero */
SW_HD bool sw_exp_gone(double x) { return sw_hi_float(x) < __int_as_float(0xC0875000); }

/* sw_pow's general case for middling x > 0 (sw_log_dd, then exp of y log x),
 * its two quotients by the same divisor in [2, 4) sharing a reciprocal; *ok
 * is cleared where the result is not that of sw_pow */
SW_HD double sw_pow_mid(double x, double y, bool *ok)
{
    const int hi = __double2hiint(x);
    const int e = (hi >> 20) - 1023;
    const double m = __hiloint2double((hi & 0x000fffff) | 0x3ff00000, __double2loint(x));
    const int i = (int)((m - 1.0) * 32.0 + 0.5);
    const double c = 1.0 + (double)i * 0.03125;
    const double num = m - c;
    const double dh = m + c;
    const double bb = dh - m;
    const double dl = (m - (dh - bb)) + (c - bb);
    const double yd = sw_rcp(dh);
    const double sh = sw_quot(num, dh, yd);
    double rem = fma(-sh, dh, num);
    rem = fma(-sh, dl, rem);
    const double sl = sw_quot(rem, dh, yd);
    const double s2 = sh * sh;
    double tq = fma(s2, sw_kc[K_ATANH_C11], sw_kc[K_ATANH_C9]);
    tq = fma(s2, tq, sw_kc[K_ATANH_C7]);
    tq = fma(s2, tq, sw_kc[K_ATANH_C5]);
    tq = fma(s2, tq, sw_kc[K_ATANH_C3]);
    const double tail = (sh * s2) * tq;
    const double l1h = 2.0 * sh;
    const double l1l = fma(2.0, sl, tail);
    const double ed = (double)e;
    const double ah = ed * sw_kc[K_LN2_HI];
    double al = fma(ed, sw_kc[K_LN2_HI], -ah);
    al = fma(ed, sw_kc[K_LN2_LO], al);
    const double ch = sw_logc_hi[i], cl = sw_logc_lo[i];
    const double s1 = ah + ch;
    const double t1 = s1 - ah;
    const double e1 = (ah - (s1 - t1)) + (ch - t1);
    const double s3 = s1 + l1h;
    const double t3 = s3 - s1;
    const double e3 = (s1 - (s3 - t3)) + (l1h - t3);
    const double low = ((al + cl) + l1l) + (e1 + e3);
    const double lh = s3 + low;
    const double ll = low - (lh - s3);
    const double th = y * lh;
    double tl = fma(y, lh, -th);
    tl = fma(y, ll, tl);
    *ok &= sw_mid_pos(x) & sw_exp_fits(th);
    return sw_exp_mid(th, tl);
}

/* sw_cos_atan for |x| < 2^400 (0x58F00000), else *ok is cleared */
SW_HD double sw_cos_atan_mid(double x, bool *ok)
{
    const double ax = fabs(x);
    const double p = ax * ax;
    const double pe = fma(ax, ax, -p);
    const double sh = 1.0 + p;
    const double bb = sh - 1.0;
    const double sl = ((1.0 - (sh - bb)) + (p - bb)) + pe;
    const double root = sw_sqrt_pos(sh);
    *ok &= sw_below(x, 0x58F00000);
    const double r0 = sw_quot(1.0, root, sw_rcp(root));
    const double q = r0 * r0;
    const double qe = fma(r0, r0, -q);
    double e = fma(-sh, q, 1.0);
    e = fma(-sh, qe, e);
    e = fma(-sl, q, e);
    return fma(r0, 0.5 * e, r0);
}
#endif

#endif /* SWEHR_IEEE_H */
