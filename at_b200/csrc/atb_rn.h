/*
 * Correctly rounded quotients and reciprocals from a reciprocal at hand.
 *
 * The exact kernels must round every division of the reference's expressions
 * as IEEE does.  Inside a magnet the divisors are 1 + delta, its rounded
 * reciprocal, their squares and numbers near one, whose reciprocals are known
 * already or one short series away, so a quotient needs no seed instruction,
 * no range test and no slow branch of its own: a product, the remainder (exact
 * in one fused operation) and one correction,
 *
 *     q0 = RN(a y),  r = b q0 - a,  q = RN(q0 - r y),
 *
 * the step proved by P. Markstein (IBM J. Res. Dev. 34, 1990: with y = RN(1/b)
 * and q0 next to a/b, q = RN(a/b)), used for a divisor known in advance as by
 * Brisebarre, Muller and Raina (IEEE Trans. Comput. 53, 2004).
 *
 * Why each use here is exact (u = 2^-53, o = RN(1 + delta), p = RN(1/o)).
 * A quotient a/b of two doubles is at least ulp(b) / (2 b) ulp(q) away from
 * any midpoint of the q grid; near a midpoint |r| is half an ulp of q times b.
 * The corrected value errs by |r| |y - 1/b| before its last rounding, so it
 * rounds as a/b does when  b^2 |y - 1/b| < ulp(b):
 *   - y = RN(1/b) (rn_div with y = p, b = o, or both scaled by two):
 *     |y - 1/b| <= ulp(y) / 2, and b^2 ulp(y) / 2 is below ulp(b) for every b
 *     in (1/2, 1) and (1, 2).
 *   - b = p, y = o (rn_div(a, p, o)): |o - 1/p| <= o^2 ulp(p) / 2, and
 *     b^2 o^2 ulp(p) / 2 = ulp(p) / 2.
 *   - b = RN(p p), y one step from RN(o o) (rn_rcp_step): within
 *     (1/2 + 2^-49) ulp of 1/b, which suffices for b > 1 and for b below
 *     1 - 2^-49; between, b = 1 - 4 i u (p = 1 - 2 i u there) has a reciprocal
 *     far from any midpoint, so y = RN(1/b).
 * The remainder is exact, or the quotient lies more than an ulp and less than
 * one and a half from q0, where rounding it in its last bit changes nothing.
 * A reciprocal's last step, y + y (1 - d y), is exact for y next to 1/d unless
 * d's significand is all ones (Markstein).  There 1/d lies just above the
 * midpoint of its neighbours and the step from the upper one is right, from
 * the lower one wrong, so the y before it is rounded upwards (rn_fma_up).
 * That may leave y an ulp and a little above 1/d where 1/d is within 2^-54 of
 * a double: far from any midpoint, and the step is right again.
 * No step may underflow or overflow: the callers bound the operands and send
 * everything else through the plain divisions.
 *
 * The functions compile for the host as well, where the CPU tests compare
 * them with the hardware's division.
 */
#ifndef ATB_RN_H
#define ATB_RN_H

#include <fenv.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define ATB_RN_FN __host__ __device__ __forceinline__
#else
#define ATB_RN_FN static inline
#endif

/* high and low words of a double's bits */
ATB_RN_FN uint32_t rn_hi(double v) {
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2hiint(v);
#else
    uint64_t b;
    memcpy(&b, &v, 8);
    return (uint32_t)(b >> 32);
#endif
}
ATB_RN_FN uint32_t rn_lo(double v) {
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2loint(v);
#else
    uint64_t b;
    memcpy(&b, &v, 8);
    return (uint32_t)b;
#endif
}

/* ---- conditions --------------------------------------------------------- */

/* v in [lo, hi) for positive bounds whose low words are zero */
ATB_RN_FN bool rn_within(double v, uint32_t lo_hi, uint32_t hi_hi) {
    return rn_hi(v) - lo_hi < hi_hi - lo_hi;
}
/* |v| below the positive bound of high word hi_hi (NaN: no) */
ATB_RN_FN bool rn_below(double v, uint32_t hi_hi) {
    return (rn_hi(v) & 0x7fffffffu) < hi_hi;
}
/* 1 + delta in a magnet without radiation, in [1/2, 2) */
ATB_RN_FN bool rn_opd_constant(double o) { return rn_within(o, 0x3fe00000u, 0x40000000u); }
/* 1 + delta at the entry of a radiating magnet, in [97/128, 5/4): the kicks
   that rn_rcp_from and rn_rcp_from_wide accept (3 x 4096 of 2^-18, 3 x 256 of
   2^-14) leave it in (0.7072, 1.4141), where its square and that of its
   reciprocal are between 1/2 and 2 */
ATB_RN_FN bool rn_opd_fits(double o) { return rn_within(o, 0x3fe84000u, 0x3ff40000u); }
/* What is left to exclude per particle are tiny nonzero values, whose
   remainders or squares would underflow: two integer instructions each, zeros
   passing.  A denormal below 2^-1042 has a zero high word and passes as well;
   rn_denormal finds it where it would matter. */
/* |v| zero or at least 2^-480 */
ATB_RN_FN bool rn_not_tiny(double v) {
    const uint32_t h = rn_hi(v);
    return h + h - 2u >= 2u * 0x21f00000u - 2u;
}
/* each of a magnet's entering coordinates zero or at least 2^-400 in size */
ATB_RN_FN bool rn_coords_fit(double x, double px, double y, double py) {
    const uint32_t a = 2u * rn_hi(x) - 2u, b = 2u * rn_hi(px) - 2u;
    const uint32_t c = 2u * rn_hi(y) - 2u, d = 2u * rn_hi(py) - 2u;
    const uint32_t ab = a < b ? a : b, cd = c < d ? c : d;
    return (ab < cd ? ab : cd) >= 2u * 0x26f00000u - 2u;
}
/* nonzero with a zero high word */
ATB_RN_FN bool rn_denormal(double v) { return 2u * rn_hi(v) == 0u && rn_lo(v) != 0u; }
/* zero or at least 2^-480 in size, and below 2^400: what a magnet's exit is
   tested for.  A quotient of values below 2^-960 may be wrong in its last
   bits.  Added to anything of ordinary size it vanishes in the rounding,
   whichever bits it has; where it does not, the sum is as tiny, and is found
   here at the exit. */
ATB_RN_FN bool rn_ordinary(double v) {
    return rn_not_tiny(v) && !rn_denormal(v) && rn_below(v, 0x58f00000u);
}

/* The domains of single operations, for the tests: the kernels need no test of
   their own for them. */
/* 1 - 2^-53, the all-ones significand next to one */
ATB_RN_FN bool rn_below_one(double v) {
    return rn_hi(v) == 0x3fefffffu && rn_lo(v) == 0xffffffffu;
}
/* divisors of rn_rcp_near: normal, below 2^1000 */
ATB_RN_FN bool rn_near_fits(double d) { return rn_within(d, 0x00100000u, 0x7e700000u); }
/* the same of divisors known to be at least 1 */
ATB_RN_FN bool rn_nearer_fits(double d) { return rn_within(d, 0x3ff00000u, 0x7e700000u); }
/* v >= 0: zero or at least 2^-860 */
ATB_RN_FN bool rn_square_fits(double v) { return rn_hi(v) - 1u >= 0x0a300000u - 1u; }

/* ---- arithmetic --------------------------------------------------------- */

/* RN(a / b) from y (see above); zeros keep the quotient's sign */
ATB_RN_FN double rn_div(double a, double b, double y) {
    const double q = a * y;
    const double r = fma(b, q, -a);
    return fma(-r, y, q);
}

/* one Newton step of the reciprocal of d */
ATB_RN_FN double rn_rcp_step(double d, double y) { return fma(fma(-d, y, 1.0), y, y); }

/* a b + c rounded upwards */
ATB_RN_FN double rn_fma_up(double a, double b, double c) {
#ifdef __CUDA_ARCH__
    return __fma_ru(a, b, c);
#else
    volatile double x = a, r;
    const int mode = fegetround();
    fesetround(FE_UPWARD);
    r = fma(x, b, c);
    fesetround(mode);
    return r;
#endif
}

/* RN(1 / o) from the reciprocal `seed` of a neighbouring number: e = 1 - o seed
   must be below 2^-18, or 2^-14 with a term more (the series drop e^3 and e^4) */
ATB_RN_FN double rn_rcp_from(double o, double seed, double* e) {
    const double d = fma(-o, seed, 1.0);
    *e = d;
    return rn_rcp_step(o, rn_fma_up(seed, fma(d, d, d), seed));
}
#define ATB_RN_SEED_HI 0x3ed00000u   /* 2^-18 */
ATB_RN_FN double rn_rcp_from_wide(double o, double seed, double* e) {
    const double d = fma(-o, seed, 1.0);
    *e = d;
    return rn_rcp_step(o, rn_fma_up(seed, fma(fma(d, d, d), d, d), seed));
}
/* its bound, by the steps that 1 + delta has to stay in range for */
ATB_RN_FN uint32_t rn_seed_wide_hi(int nsteps) {
    return nsteps <= 256 ? 0x3f100000u : ATB_RN_SEED_HI;   /* 2^-14 */
}

/* 1 / d to 20 bits (on the host, for the tests, the quotient's high word) */
ATB_RN_FN double rn_estimate(double d) {
    double y;
#ifdef __CUDA_ARCH__
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
#else
    uint64_t b;
    y = 1.0 / d;
    memcpy(&b, &y, 8);
    b &= 0xffffffff00000000ull;
    memcpy(&y, &b, 8);
#endif
    return y;
}

/* RN(1 / d): the estimate's residue in a geometric series to the second power
   (the third is below 2^-54 for an estimate of 18 bits), then the exact step */
ATB_RN_FN double rn_rcp_near(double d) {
    const double y = rn_estimate(d);
    const double r = fma(-d, y, 1.0);
    return rn_rcp_step(d, rn_fma_up(y, fma(r, r, r), y));
}
ATB_RN_FN double rn_rcp_nearer(double d) { return rn_rcp_near(d); }

#endif /* ATB_RN_H */
