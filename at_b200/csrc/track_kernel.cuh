/*
 * The persistent multi-turn tracking kernel.
 *
 * One thread owns one particle's (x, px, y, py, delta, ct) in registers for
 * all the turns of a launch.  A block walks the lattice program (the flat
 * element table of atb_table.h) segment by segment: each segment is copied
 * from global memory into shared memory by the bulk-copy (TMA) engine,
 * double-buffered behind an mbarrier, and every element's parameters are then
 * read from shared memory as warp-uniform broadcasts.  When the whole table
 * fits in one buffer it is loaded once per block and stays resident.
 *
 * The turn/element loop, the refpts snapshots and the loss rule restate the
 * reference engine (pyat/at.c:596-654, checkiflost :115-139, setlost
 * :142-161); the per-element bodies restate the pass methods (see
 * atb_physics.cuh).  This header is compiled twice, once per arithmetic mode
 * (ATB_FAST = 0 / 1), into distinct kernel symbols.
 */
#ifndef ATB_TRACK_KERNEL_CUH
#define ATB_TRACK_KERNEL_CUH

#include <cstdint>
#include <type_traits>
#include "atb_physics.cuh"
#include "atb_integrators.h"
#include "atb_kernel_api.h"

#ifndef ATB_FAST
#error "define ATB_FAST to 0 or 1"
#endif

/* the tracking kernels this unit instantiates (each takes a minute to
   compile, so the build gives each its own unit); the derivative units take
   none */
#define ATB_KERNEL_BASE 1
#define ATB_KERNEL_GEN 2
#define ATB_KERNEL_SERVE 4
#define ATB_KERNEL_NP2 8
#ifdef ATB_NO_TRACK_KERNEL
#define ATB_KERNELS 0
#endif
#ifndef ATB_KERNELS
#define ATB_KERNELS (ATB_KERNEL_BASE | ATB_KERNEL_GEN | ATB_KERNEL_SERVE | ATB_KERNEL_NP2)
#endif

#define ATB_CAT2(a, b) a##b
#define ATB_CAT(a, b) ATB_CAT2(a, b)
#if ATB_FAST
#define ATB_KSUFFIX _fast
#else
#define ATB_KSUFFIX _exact
#endif

namespace atb {

constexpr bool kFast = (ATB_FAST != 0);

/* ---------------- shared-memory staging (bulk copy + mbarrier) ---------- */

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
                 : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile(
        "mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
        "r"(bytes)
        : "memory");
}

/* global -> shared bulk copy into this CTA's own shared memory, completion
 * signalled on the mbarrier; the source is always this GPU's own memory */
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes,
                                         uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

/* Bounded wait: gives up after ATB_WAIT_NS nanoseconds and reports it. */
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    while (true) {
        if (mbar_try_wait(bar, parity)) return true;
        if (global_ns() - t0 > ATB_WAIT_NS) return false;
    }
}

/* ---------------- record access ------------------------------------------ */

struct Rec {
    const double* p;
    uint64_t hdr;
    uint64_t opt;
    __device__ __forceinline__ int op() const { return (int)((hdr >> ATB_H_OP_SHIFT) & ATB_H_OP_MASK); }
    __device__ __forceinline__ int mo() const { return (int)((hdr >> ATB_H_MO_SHIFT) & ATB_H_MO_MASK); }
    __device__ __forceinline__ uint32_t flags() const { return (uint32_t)((hdr >> ATB_H_FL_SHIFT) & ATB_H_FL_MASK); }
    __device__ __forceinline__ int nsteps() const { return (int)((hdr >> ATB_H_NS_SHIFT) & ATB_H_NS_MASK); }
    __device__ __forceinline__ int len() const { return (int)((hdr >> ATB_H_LEN_SHIFT) & ATB_H_LEN_MASK); }
    __device__ __forceinline__ const double* blk(int slot) const {
        uint32_t o = (uint32_t)((opt >> (slot * ATB_OPT_BITS)) & ATB_OPT_MASK);
        return o ? p + o : nullptr;
    }
    __device__ __forceinline__ double f(int w) const { return p[w]; }
};

/* ---------------- misalignment / aperture wrappers ----------------------- */

#define ATB_OPT_FIELD(slot) ((uint64_t)ATB_OPT_MASK << ((slot) * ATB_OPT_BITS))
#define ATB_OPT_APERTURES (ATB_OPT_FIELD(ATB_OPT_RAP) | ATB_OPT_FIELD(ATB_OPT_EAP))

static __device__ __noinline__ P6 mult_dense_call(P6 r, const double* m) {
    mult_dense(r, m);
    return r;
}
/* whether (x, y) is outside an element's apertures (null: none) */
static __device__ __noinline__ bool outside_call(double x, double y, const double* rect,
                                                 const double* ellip) {
    P6 r;
    r.x = x;
    r.y = y;
    r.ct = 0.0;
    if (rect) check_rect(r, rect);
    if (ellip) check_ellip(r, ellip);
    return r.ct != 0.0;
}

/* CALL: the rare forms out of line */
template <bool CALL = false, class T>
__device__ __forceinline__ void misalign_rotation(P6T<T>& r, const double* m, bool dense) {
    if constexpr (CALL) {
        if (dense) r = mult_dense_call(r, m);
        else mult_tilt(r, m);
    } else {
        mult_r(r, m, dense);
    }
}

/* The usual misalignment, a shift and a rotation of the x/y planes: one branch,
 * and the fourteen words (16-byte aligned blocks) asked for at once.  One by
 * one, each branch waited for its own words: 375 cycles a warp and magnet with
 * 16 warps on an SM, 208 so. */
struct ShiftTilt {
    double2 t[3], m[4];
};
__device__ __forceinline__ bool shift_tilt(const Rec& e, int shift, int rot, uint32_t dense,
                                           ShiftTilt& w) {
    const uint32_t ot = (uint32_t)((e.opt >> (shift * ATB_OPT_BITS)) & ATB_OPT_MASK);
    const uint32_t om = (uint32_t)((e.opt >> (rot * ATB_OPT_BITS)) & ATB_OPT_MASK);
    if (ot == 0u || om == 0u || ((ot | om) & 1u) || (e.flags() & dense)) return false;
    const double2* pt = reinterpret_cast<const double2*>(e.p + ot);
    const double2* pm = reinterpret_cast<const double2*>(e.p + om);
#pragma unroll
    for (int i = 0; i < 3; ++i) w.t[i] = pt[i];
#pragma unroll
    for (int i = 0; i < 4; ++i) w.m[i] = pm[i];
    return true;
}
__device__ __forceinline__ void shift(P6& r, const ShiftTilt& w) {
    const double t[6] = {w.t[0].x, w.t[0].y, w.t[1].x, w.t[1].y, w.t[2].x, w.t[2].y};
    add_t(r, t);
}
__device__ __forceinline__ void tilt(P6& r, const ShiftTilt& w) {
    const double m[8] = {w.m[0].x, w.m[0].y, w.m[1].x, w.m[1].y,
                         w.m[2].x, w.m[2].y, w.m[3].x, w.m[3].y};
    mult_tilt(r, m);
}

template <bool CALL = false, class T>
__device__ __forceinline__ void entrance_misalign(P6T<T>& r, const Rec& e) {
    if constexpr (CALL) {
        ShiftTilt w;
        if (shift_tilt(e, ATB_OPT_T1, ATB_OPT_R1, ATB_F_R1_DENSE, w)) {
            shift(r, w);
            tilt(r, w);
            return;
        }
    }
    const uint32_t fl = e.flags();
    if (const double* t1 = e.blk(ATB_OPT_T1)) add_t(r, t1);
    if (const double* r1 = e.blk(ATB_OPT_R1))
        misalign_rotation<CALL>(r, r1, fl & ATB_F_R1_DENSE);
}

template <bool CALL = false, class T>
__device__ __forceinline__ void apertures(P6T<T>& r, const Rec& e) {
    if constexpr (CALL) {
        if (__builtin_expect((e.opt & ATB_OPT_APERTURES) != 0, 0))
            if (outside_call(r.x, r.y, e.blk(ATB_OPT_RAP), e.blk(ATB_OPT_EAP))) r.ct = inf_d();
    } else {
        if (const double* ra = e.blk(ATB_OPT_RAP)) check_rect(r, ra);
        if (const double* ea = e.blk(ATB_OPT_EAP)) check_ellip(r, ea);
    }
}

template <bool CALL = false, class T>
__device__ __forceinline__ void exit_misalign(P6T<T>& r, const Rec& e) {
    if constexpr (CALL) {
        ShiftTilt w;
        if (shift_tilt(e, ATB_OPT_T2, ATB_OPT_R2, ATB_F_R2_DENSE, w)) {
            tilt(r, w);
            shift(r, w);
            return;
        }
    }
    const uint32_t fl = e.flags();
    if (const double* r2 = e.blk(ATB_OPT_R2))
        misalign_rotation<CALL>(r, r2, fl & ATB_F_R2_DENSE);
    if (const double* t2 = e.blk(ATB_OPT_T2)) add_t(r, t2);
}

/* ---------------- pass methods ------------------------------------------- */

/* A differentiated strength (derivative kernels only): PolynomB[k] of the
 * element is replaced by v and, on dual numbers, carried as the last
 * derivative direction.  The tracking kernels pass k = -1. */
struct Param {
    int k;        /* coefficient order, -1: none */
    double v;
};

/* the quadrupole-fringe gradient b1 = PolynomB[1], seeded when it is the
 * differentiated strength */
template <class T>
__device__ __forceinline__ T fringe_b1(const Rec& e, const Param& pm) {
    T b1 = e.f(ATB_SM_B1);
    if constexpr (is_dual<T>::value) {
        if (pm.k == 1) {
            b1.v = pm.v;
            b1.d[sizeof(b1.d) / sizeof(double) - 1] = 1.0;
        }
    } else {
        if (pm.k == 1) b1 = pm.v;
    }
    return b1;
}

/* 1/(1+delta) of the momentum it was last asked for.  delta changes only in
 * cavities and radiating kicks (whose loops leave the new reciprocal here),
 * so drifts and magnets mostly find theirs without a division.  The dual
 * numbers of the derivative kernels divide every time. */
struct Recip {
    double dp, pn;
    __device__ __forceinline__ Recip() : dp(nan_d()), pn(0.0) {}
};
template <class T>
struct NoRecip {};
template <class T>
using RecipOf = typename std::conditional<is_dual<T>::value, NoRecip<T>, Recip>::type;

__device__ __forceinline__ double opd_rcp(Recip& c, double dp) {
    if (dp != c.dp) {
        c.dp = dp;
        c.pn = 1.0 / (1.0 + dp);
    }
    return c.pn;
}
template <class T>
__device__ __forceinline__ T opd_rcp(NoRecip<T>&, const T& dp) {
    return 1.0 / (1.0 + dp);
}

/* The integration steps of a thick multipole under integrator id
 * e.f(ATB_SM_INTEG) (1-6, atb_integrators.h), step SL = e.f(ATB_SM_SL): per
 * step, for each stage a drift of SL*c[i] and a kick of SL*d[i], skipping zero
 * coefficients.  The drift and kick are the ones the Forest-Ruth steps use:
 * fastdrift with the entrance 1/(1+delta) in plain magnets (pnorm: the
 * entrance L2 x 1/(1+delta) with the table's L2 word set to 1.0), the
 * radiating drift and kicks otherwise (the angle-carrying forms in the fast
 * kernels). */
template <int NP, bool BEND, bool RAD, class PL, class T>
__device__ __forceinline__ void multipole_steps_generic(P6T<T>* r, const Rec& e, const PL& pl,
                                                        const T* pnorm, double irho, int ns) {
    const double SL = e.f(ATB_SM_SL);
    int id = (int)e.f(ATB_SM_INTEG);
    if (id < 1 || id >= ATB_INTEG_COUNT) id = 4;   /* the host writes 1-6 only */
    const AtbInteg& ig = atb_integ[id];
    if (RAD) {
        const double radc = e.f(ATB_SM_RADC);
        if constexpr (kFast && !is_dual<T>::value) {
            if (ns <= 0) return;
            RadAngles a[NP];
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                const double pn = 1.0 / (1.0 + r[k].dp);
                a[k] = RadAngles{r[k].px * pn, r[k].py * pn, 0.0, 1.0 + r[k].dp};
            }
            for (int m = 0; m < ns; ++m) {
                for (int i = 0; i < ig.n; ++i) {
                    if (ig.c[i] != 0.0) {
                        const double ld = SL * ig.c[i];
#pragma unroll
                        for (int k = 0; k < NP; ++k) rad_drift_fast(r[k], a[k], ld, 0.5 * ld);
                    }
                    if (ig.d[i] != 0.0) {
                        const double lk = SL * ig.d[i];
#pragma unroll
                        for (int k = 0; k < NP; ++k) {
                            if (BEND) bnd_kick_rad_fast(r[k], a[k], pl, lk, irho, lk * irho, radc * lk);
                            else str_kick_rad_fast(r[k], a[k], pl, lk, radc * lk);
                        }
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                r[k].px = a[k].xp * a[k].opd;
                r[k].py = a[k].yp * a[k].opd;
            }
        } else {
            T pn[NP];   /* 1/(1+delta) as last evaluated, as in the steps below */
#pragma unroll
            for (int k = 0; k < NP; ++k) pn[k] = 1.0 / (1.0 + r[k].dp);
            for (int m = 0; m < ns; ++m) {
                for (int i = 0; i < ig.n; ++i) {
                    if (ig.c[i] != 0.0) {
                        const double ld = SL * ig.c[i];
#pragma unroll
                        for (int k = 0; k < NP; ++k) diff_drift_pn(r[k], ld, pn[k]);
                    }
                    if (ig.d[i] != 0.0) {
                        const double lk = SL * ig.d[i];
#pragma unroll
                        for (int k = 0; k < NP; ++k) {
                            if (BEND) bnd_kick_rad_pn(r[k], pl, lk, irho, lk * irho, radc, pn[k]);
                            else str_kick_rad_pn(r[k], pl, lk, radc, pn[k]);
                        }
                    }
                }
            }
        }
    } else {
        T h[NP];
#pragma unroll
        for (int k = 0; k < NP; ++k) h[k] = kFast ? T(0.5 / (1.0 + r[k].dp)) : T(0.0);
        for (int m = 0; m < ns; ++m) {
            for (int i = 0; i < ig.n; ++i) {
                if (ig.c[i] != 0.0) {
                    const double ld = SL * ig.c[i];
#pragma unroll
                    for (int k = 0; k < NP; ++k) {
                        const T nl = ld * pnorm[k];
                        fastdrift<kFast>(r[k], nl, kFast ? T(nl * h[k]) : T(0.0));
                    }
                }
                if (ig.d[i] != 0.0) {
                    const double lk = SL * ig.d[i];
#pragma unroll
                    for (int k = 0; k < NP; ++k) {
                        if (BEND) bndthinkick(r[k], pl, lk, irho, lk * irho);
                        else strthinkick(r[k], pl, lk);
                    }
                }
            }
        }
    }
}

/* The Forest-Ruth steps of a thick multipole by the reference's plain
 * expressions (StrMPoleSymplectic4Pass.c:73-93 and the Bnd and Rad variants);
 * nl1, nl2: the drift lengths of the non-radiating variants, scaled by
 * 1/(1+delta) of the element's entry. */
template <int NP, bool BEND, bool RAD, class PL, class T>
__device__ __forceinline__ void multipole_steps_plain(P6T<T>* r, const Rec& e, const PL& pl,
                                                      const T* nl1, const T* nl2, double irho,
                                                      int ns) {
    const double K1 = e.f(ATB_SM_K1), K2 = e.f(ATB_SM_K2);
    const double k1i = BEND ? e.f(ATB_BM_K1IRHO) : 0.0, k2i = BEND ? e.f(ATB_BM_K2IRHO) : 0.0;
    if (RAD) {
        const double L1 = e.f(ATB_SM_L1), L2 = e.f(ATB_SM_L2), radc = e.f(ATB_SM_RADC);
        /* pn: 1/(1+delta) as the reference last evaluated it (it changes
           only in a kick's energy loss, and the kick hands it on) */
        T pn[NP];
#pragma unroll
        for (int k = 0; k < NP; ++k) pn[k] = 1.0 / (1.0 + r[k].dp);
        for (int m = 0; m < ns; ++m) {
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                diff_drift_pn(r[k], L1, pn[k]);
                if (BEND) bnd_kick_rad_pn(r[k], pl, K1, irho, k1i, radc, pn[k]);
                else str_kick_rad_pn(r[k], pl, K1, radc, pn[k]);
                diff_drift_pn(r[k], L2, pn[k]);
                if (BEND) bnd_kick_rad_pn(r[k], pl, K2, irho, k2i, radc, pn[k]);
                else str_kick_rad_pn(r[k], pl, K2, radc, pn[k]);
                diff_drift_pn(r[k], L2, pn[k]);
                if (BEND) bnd_kick_rad_pn(r[k], pl, K1, irho, k1i, radc, pn[k]);
                else str_kick_rad_pn(r[k], pl, K1, radc, pn[k]);
                diff_drift_pn(r[k], L1, pn[k]);
            }
        }
    } else {
        for (int m = 0; m < ns; ++m) {
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                fastdrift<false>(r[k], nl1[k], T(0.0));
                if (BEND) bndthinkick(r[k], pl, K1, irho, k1i); else strthinkick(r[k], pl, K1);
                fastdrift<false>(r[k], nl2[k], T(0.0));
                if (BEND) bndthinkick(r[k], pl, K2, irho, k2i); else strthinkick(r[k], pl, K2);
                fastdrift<false>(r[k], nl2[k], T(0.0));
                if (BEND) bndthinkick(r[k], pl, K1, irho, k1i); else strthinkick(r[k], pl, K1);
                fastdrift<false>(r[k], nl1[k], T(0.0));
            }
        }
    }
}

/* The same out of line, for the rare magnet whose operands leave the range of
 * multipole_steps_rn. */
template <bool BEND, bool RAD>
__device__ __noinline__ P6 multipole_steps_call(P6 r, Rec e, Param pm, double nl1, double nl2) {
    const int mo = e.mo();
    const double* A = e.p + (BEND ? ATB_BM_POLY : ATB_SM_POLY);
    Poly<-1> pl;
    pl.load(A, A + mo + 1, mo);
    if (pm.k >= 0) pl.set_param(pm.k, pm.v);
    multipole_steps_plain<1, BEND, RAD>(&r, e, pl, &nl1, &nl2, BEND ? e.f(ATB_BM_IRHO) : 0.0,
                                        e.nsteps());
    return r;
}

/* multipole_steps_plain on doubles in the exact kernels, with the divisions
 * of atb_rn.h: the same IEEE results, straight-line code in the step loop.
 * The divisions bounded these loops: about nine FP64 instructions each, a
 * seed on the XU pipe and a branch to a slow path that ended the block the
 * compiler could interleave (a sextupole step without radiation took a lone
 * warp 631 cycles and takes 271, one with radiation 1,886 and 724).  The last drift
 * of a step and the first of the next have the same length, momenta and
 * 1/(1+delta), hence the same increments: they are computed once and added
 * twice.
 * Conditions belong outside the loop, where they do not wait for the kicks:
 * with the path factor, the angles and the roundings next to one tested in
 * every kick a turn of the large ring took 5.2 ms for one warp an SM and 40.9
 * for 300,000 particles, with the largest loss alone kept there and the rest
 * at the ends 4.35 and 34.5.  Out of range are energy losses above 2^-14 in
 * one kick of a bend (2^-18 with more than 256 steps), 2^-18 in a straight
 * magnet, 1 + delta outside [97/128, 5/4) ([1/2, 2) without radiation), and
 * what overflows: particles about to be lost.  Such a magnet is tracked again
 * from its entry; one that is out of range there takes a single step first. */
template <int NP, bool BEND, bool RAD, class PL>
__device__ __forceinline__ void multipole_steps_rn(P6* r, Recip* c, const Rec& e, const PL& pl,
                                                   const Param& pm, const double* pb,
                                                   const double* nl1, const double* nl2,
                                                   double irho, int ns) {
    if (ns <= 0) return;
    const double K1 = e.f(ATB_SM_K1), K2 = e.f(ATB_SM_K2);
    const double k1i = BEND ? e.f(ATB_BM_K1IRHO) : 0.0, k2i = BEND ? e.f(ATB_BM_K2IRHO) : 0.0;
    P6 in[NP];
    bool ok[NP];
    DriftInc d1[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) {
        in[k] = r[k];
        ok[k] = (e.flags() & ATB_F_RN) &&
                (RAD ? rn_opd_fits(1.0 + r[k].dp) &&
                           rn_coords_fit(r[k].x, r[k].px, r[k].y, r[k].py)
                     : rn_opd_constant(1.0 + r[k].dp));
    }
    /* out of range already: a single step here, for nothing */
    int m = ns;
#pragma unroll
    for (int k = 0; k < NP; ++k)
        if (ok[k]) m = 1;
    if (RAD) {
        const double L1 = e.f(ATB_SM_L1), L2 = e.f(ATB_SM_L2), radc = e.f(ATB_SM_RADC);
        double o[NP], pn[NP];
        uint32_t loss[NP];             /* the largest kick's, its high word */
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            o[k] = 1.0 + r[k].dp;
            pn[k] = opd_rcp(c[k], r[k].dp);
            loss[k] = 0u;
            d1[k] = drift_rad_inc(r[k], L1, pn[k]);
            add_drift_rad(r[k], d1[k]);
        }
        for (;; ++m) {
#pragma unroll
            for (int k = 0; k < NP; ++k)
                kick_rad_rn<BEND>(r[k], pl, K1, irho, k1i, radc, o[k], pn[k], loss[k]);
#pragma unroll
            for (int k = 0; k < NP; ++k) add_drift_rad(r[k], drift_rad_inc(r[k], L2, pn[k]));
#pragma unroll
            for (int k = 0; k < NP; ++k)
                kick_rad_rn<BEND>(r[k], pl, K2, irho, k2i, radc, o[k], pn[k], loss[k]);
#pragma unroll
            for (int k = 0; k < NP; ++k) add_drift_rad(r[k], drift_rad_inc(r[k], L2, pn[k]));
#pragma unroll
            for (int k = 0; k < NP; ++k)
                kick_rad_rn<BEND>(r[k], pl, K1, irho, k1i, radc, o[k], pn[k], loss[k]);
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                d1[k] = drift_rad_inc(r[k], L1, pn[k]);
                add_drift_rad(r[k], d1[k]);
            }
            if (m == ns) break;
#pragma unroll
            for (int k = 0; k < NP; ++k) add_drift_rad(r[k], d1[k]);
        }
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            ok[k] &= loss[k] < (BEND ? rn_seed_wide_hi(ns) : ATB_RN_SEED_HI) &&
                     rn_ordinary(r[k].x) && rn_ordinary(r[k].px) && rn_ordinary(r[k].y) &&
                     rn_ordinary(r[k].py);
            c[k].dp = r[k].dp;
            c[k].pn = pn[k];
        }
    } else {
        double od2[NP], hp[NP];
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            od2[k] = 2.0 * (1.0 + r[k].dp);
            hp[k] = 0.5 * pb[k];
            d1[k] = fastdrift_inc(r[k], nl1[k], od2[k], hp[k]);
            add_drift(r[k], d1[k]);
        }
        for (;; ++m) {
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                if (BEND) bndthinkick(r[k], pl, K1, irho, k1i); else strthinkick(r[k], pl, K1);
            }
#pragma unroll
            for (int k = 0; k < NP; ++k)
                add_drift(r[k], fastdrift_inc(r[k], nl2[k], od2[k], hp[k]));
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                if (BEND) bndthinkick(r[k], pl, K2, irho, k2i); else strthinkick(r[k], pl, K2);
            }
#pragma unroll
            for (int k = 0; k < NP; ++k)
                add_drift(r[k], fastdrift_inc(r[k], nl2[k], od2[k], hp[k]));
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                if (BEND) bndthinkick(r[k], pl, K1, irho, k1i); else strthinkick(r[k], pl, K1);
            }
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                d1[k] = fastdrift_inc(r[k], nl1[k], od2[k], hp[k]);
                add_drift(r[k], d1[k]);
            }
            if (m == ns) break;
#pragma unroll
            for (int k = 0; k < NP; ++k) add_drift(r[k], d1[k]);
        }
        /* an overflow anywhere has reached ct; it is also where the
           quotients have gone */
#pragma unroll
        for (int k = 0; k < NP; ++k) ok[k] &= rn_ordinary(r[k].ct);
    }
#pragma unroll
    for (int k = 0; k < NP; ++k)
        if (!ok[k]) {
            r[k] = multipole_steps_call<BEND, RAD>(in[k], e, pm, nl1[k], nl2[k]);
            c[k] = Recip();
        }
}

/* The fast kernels' radiating steps.  A step's last drift and the first of
 * the next share angles and increments. */
template <int NP, bool BEND, class PL>
__device__ __forceinline__ void rad_steps_fast(P6* r, Recip* c, const Rec& e, const PL& pl,
                                               double irho, int ns) {
    const double K1 = e.f(ATB_SM_K1), K2 = e.f(ATB_SM_K2);
    const double k1i = BEND ? e.f(ATB_BM_K1IRHO) : 0.0, k2i = BEND ? e.f(ATB_BM_K2IRHO) : 0.0;
    const double L1 = e.f(ATB_SM_L1), L2 = e.f(ATB_SM_L2), radc = e.f(ATB_SM_RADC);
    const double rk1 = radc * K1, rk2 = radc * K2, h1 = 0.5 * L1, h2 = 0.5 * L2;
    RadAngles a[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) {
        const double pn = opd_rcp(c[k], r[k].dp);
        a[k] = RadAngles{r[k].px * pn, r[k].py * pn, 0.0, 1.0 + r[k].dp};
        rad_drift_fast(r[k], a[k], L1, h1);
    }
    for (int m = 1;; ++m) {
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            if (BEND) bnd_kick_rad_fast(r[k], a[k], pl, K1, irho, k1i, rk1);
            else str_kick_rad_fast(r[k], a[k], pl, K1, rk1);
        }
#pragma unroll
        for (int k = 0; k < NP; ++k) rad_drift_fast(r[k], a[k], L2, h2);
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            if (BEND) bnd_kick_rad_fast(r[k], a[k], pl, K2, irho, k2i, rk2);
            else str_kick_rad_fast(r[k], a[k], pl, K2, rk2);
        }
#pragma unroll
        for (int k = 0; k < NP; ++k) rad_drift_fast(r[k], a[k], L2, h2);
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            if (BEND) bnd_kick_rad_fast(r[k], a[k], pl, K1, irho, k1i, rk1);
            else str_kick_rad_fast(r[k], a[k], pl, K1, rk1);
        }
#pragma unroll
        for (int k = 0; k < NP; ++k) rad_drift_fast(r[k], a[k], L1, h1);
        if (m == ns) break;
#pragma unroll
        for (int k = 0; k < NP; ++k) rad_drift_again(r[k], a[k], L1, h1);
    }
#pragma unroll
    for (int k = 0; k < NP; ++k) {
        r[k].px = a[k].xp * a[k].opd;
        r[k].py = a[k].yp * a[k].opd;
    }
}

/* The fast kernels' steps. */
template <int NP, bool BEND, bool RAD, class PL>
__device__ __forceinline__ void multipole_steps_fast(P6* r, Recip* c, const Rec& e, const PL& pl,
                                                     const double* nl1, const double* nl2,
                                                     double irho, int ns) {
    if (ns <= 0) return;
    if (RAD) {
        rad_steps_fast<NP, BEND>(r, c, e, pl, irho, ns);
    } else {
        const double K1 = e.f(ATB_SM_K1), K2 = e.f(ATB_SM_K2);
        const double k1i = BEND ? e.f(ATB_BM_K1IRHO) : 0.0, k2i = BEND ? e.f(ATB_BM_K2IRHO) : 0.0;
        double c1[NP], c2[NP];
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            const double h = 0.5 * opd_rcp(c[k], r[k].dp);
            c1[k] = nl1[k] * h;
            c2[k] = nl2[k] * h;
        }
        for (int m = 0; m < ns; ++m) {
#pragma unroll
            for (int k = 0; k < NP; ++k) fastdrift<kFast>(r[k], nl1[k], c1[k]);
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                if (BEND) bndthinkick(r[k], pl, K1, irho, k1i); else strthinkick(r[k], pl, K1);
            }
#pragma unroll
            for (int k = 0; k < NP; ++k) fastdrift<kFast>(r[k], nl2[k], c2[k]);
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                if (BEND) bndthinkick(r[k], pl, K2, irho, k2i); else strthinkick(r[k], pl, K2);
            }
#pragma unroll
            for (int k = 0; k < NP; ++k) fastdrift<kFast>(r[k], nl2[k], c2[k]);
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                if (BEND) bndthinkick(r[k], pl, K1, irho, k1i); else strthinkick(r[k], pl, K1);
            }
#pragma unroll
            for (int k = 0; k < NP; ++k) fastdrift<kFast>(r[k], nl1[k], c1[k]);
        }
    }
}

/* The integration steps with the coefficients of MaxOrder MO in registers
 * (-1: read from the table on every kick). */
template <int NP, int MO, bool BEND, bool RAD, bool SKEW>
__device__ __forceinline__ void multipole_steps_mo(P6* r, Recip* c, const Rec& e, const Param& pm,
                                                   const double* pb, const double* nl1,
                                                   const double* nl2, double irho, int ns) {
    const int mo = e.mo();
    const double* A = e.p + (BEND ? ATB_BM_POLY : ATB_SM_POLY);
    Poly<MO, SKEW> pl;
    pl.load(A, A + mo + 1, mo);
    if (pm.k >= 0) pl.set_param(pm.k, pm.v);
    if constexpr (kFast) multipole_steps_fast<NP, BEND, RAD>(r, c, e, pl, nl1, nl2, irho, ns);
    else multipole_steps_rn<NP, BEND, RAD>(r, c, e, pl, pm, pb, nl1, nl2, irho, ns);
}

template <int NP, bool BEND, bool RAD, bool INTEG, class T>
__device__ __forceinline__ void multipole_steps(P6T<T>* r, RecipOf<T>* c, const Rec& e,
                                                const Param& pm, const double* pb, const T* nl1,
                                                const T* nl2, double irho, int ns) {
    if constexpr (is_dual<T>::value) {
        /* one generic instance for the tangent kernel keeps its size sane */
        const int mo = e.mo();
        const double* A = e.p + (BEND ? ATB_BM_POLY : ATB_SM_POLY);
        Poly<-1> pl;
        pl.load(A, A + mo + 1, mo);
        if (pm.k >= 0) pl.set_param(pm.k, pm.v);
        multipole_steps_plain<NP, BEND, RAD>(r, e, pl, nl1, nl2, irho, ns);
    } else if constexpr (INTEG) {
        /* another integrator of the GPU call: steps of SL*c[i] drift and
           SL*d[i] kick (atgpu/SymplecticIntegrator.cpp:140-171) */
        const int mo = e.mo();
        const double* A = e.p + (BEND ? ATB_BM_POLY : ATB_SM_POLY);
        Poly<-1> pl;
        pl.load(A, A + mo + 1, mo);
        if (pm.k >= 0) pl.set_param(pm.k, pm.v);
        multipole_steps_generic<NP, BEND, RAD>(r, e, pl, nl2, irho, ns);
    } else {
#define ATB_STEPS(MO, SKEW) \
    multipole_steps_mo<NP, MO, BEND, RAD, SKEW>(r, c, e, pm, pb, nl1, nl2, irho, ns)
        /* upright magnets' fields without the zero skew terms; the loops that
           most magnets run first, for the compiler to lay them side by side */
        const bool upright = e.flags() & ATB_F_NOSKEW;
        const int mo = e.mo();
        if (__builtin_expect(upright && mo == 1, 1)) {
            ATB_STEPS(1, false);
        } else if (__builtin_expect(upright && mo == 2, 1)) {
            ATB_STEPS(2, false);
        } else if (__builtin_expect(upright && mo == 3, 1)) {
            ATB_STEPS(3, false);
        } else {
            switch (mo) {
                case 0: ATB_STEPS(0, true); break;
                case 1: ATB_STEPS(1, true); break;
                case 2: ATB_STEPS(2, true); break;
                case 3: ATB_STEPS(3, true); break;
                default: ATB_STEPS(-1, true); break;
            }
        }
#undef ATB_STEPS
    }
}

/* StrMPoleSymplectic4Pass.c:29-109, BndMPoleSymplectic4Pass.c:38-129,
 * StrMPoleSymplectic4RadPass.c:30-115, BndMPoleSymplectic4RadPass.c:39-128.
 * NP particles of one thread pass the element together: every per-particle
 * step is an unrolled loop over them, so in the step loop their drifts and
 * kicks form one straight-line block whose independent chains the compiler
 * interleaves (NP = 2), while the element's parameters are read once.  Each
 * particle sees the same operations as alone (NP = 1).  The entrance and exit
 * are outside the choice of the step loop: one copy per pass method, which a
 * warp walking the lattice finds in the instruction cache.  LEAN: the form for
 * elements without field scaling and quadrupole fringes, with dense rotations
 * and apertures out of line. */
template <int NP, bool BEND, bool RAD, bool INTEG = false, bool LEAN = false, class T>
__device__ __forceinline__ void pass_multipole_n(P6T<T>* r, RecipOf<T>* c, const Rec& e,
                                                 const Param& pm) {
    const uint32_t fl = e.flags();
    double pb[NP];             /* 1/(1+delta) in the body of a plain magnet */
    T nl1[NP], nl2[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) {
        if (!LEAN && (fl & ATB_F_SCALING)) change_pref<kFast>(r[k], e.f(ATB_SM_SCALE));
        pb[k] = 0.0;
        nl1[k] = 0.0;
        nl2[k] = 0.0;
        if (!RAD) {
            T p_norm = opd_rcp(c[k], r[k].dp);
            pb[k] = val(p_norm);
            nl1[k] = e.f(ATB_SM_L1) * p_norm;
            nl2[k] = e.f(ATB_SM_L2) * p_norm;
        }
        if (e.opt) {
            const double dp0 = val(r[k].dp);
            entrance_misalign<LEAN>(r[k], e);
            /* a shift or a dense rotation may change delta */
            if (!RAD && val(r[k].dp) != dp0) pb[k] = 1.0 / (1.0 + val(r[k].dp));
            apertures<LEAN>(r[k], e);
        }
    }
    double irho = 0.0;
    if (BEND) {
        irho = e.f(ATB_BM_IRHO);
        const int m_in = (int)((fl >> ATB_F_BM_IN_SHIFT) & ATB_F_BM_MASK);
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            if (RAD)
                edge_fringe_rad<kFast>(r[k], irho, e.f(ATB_BM_EIN), e.f(ATB_BM_FCIN),
                                       e.f(ATB_BM_FXIN), e.f(ATB_BM_FYIN), m_in,
                                       fl & ATB_F_FC0_IN, 1.0);
            else
                edge_fringe<kFast>(r[k], irho, e.f(ATB_BM_EIN), e.f(ATB_BM_FCIN),
                                   e.f(ATB_BM_FXIN), e.f(ATB_BM_FYIN), m_in, fl & ATB_F_FC0_IN,
                                   1.0);
        }
    }
    if (!LEAN && (fl & ATB_F_FQ_IN)) {
        const T b1 = fringe_b1<T>(e, pm);
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            if (fl & ATB_F_FQ_IN_LIN) {
                const double* fm = e.blk(ATB_OPT_FRINGE);
                lin_fringe_map(r[k], fm);
                quad_fringe<kFast>(r[k], b1, true);
                lin_fringe_map(r[k], fm + 8);
            } else {
                quad_fringe<kFast>(r[k], b1, true);
            }
        }
    }
    multipole_steps<NP, BEND, RAD, INTEG>(r, c, e, pm, pb, nl1, nl2, irho, e.nsteps());
    if (!LEAN && (fl & ATB_F_FQ_OUT)) {
        const T b1 = fringe_b1<T>(e, pm);
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            if (fl & ATB_F_FQ_OUT_LIN) {
                const double* fm = e.blk(ATB_OPT_FRINGE);
                lin_fringe_map(r[k], fm + 16);
                quad_fringe<kFast>(r[k], b1, false);
                lin_fringe_map(r[k], fm + 24);
            } else {
                quad_fringe<kFast>(r[k], b1, false);
            }
        }
    }
    const int m_out = (int)((fl >> ATB_F_BM_OUT_SHIFT) & ATB_F_BM_MASK);
#pragma unroll
    for (int k = 0; k < NP; ++k) {
        if (BEND) {
            if (RAD)
                edge_fringe_rad<kFast>(r[k], irho, e.f(ATB_BM_EOUT), e.f(ATB_BM_FCOUT),
                                       e.f(ATB_BM_FXOUT), e.f(ATB_BM_FYOUT), m_out,
                                       fl & ATB_F_FC0_OUT, -1.0);
            else
                edge_fringe<kFast>(r[k], irho, e.f(ATB_BM_EOUT), e.f(ATB_BM_FCOUT),
                                   e.f(ATB_BM_FXOUT), e.f(ATB_BM_FYOUT), m_out,
                                   fl & ATB_F_FC0_OUT, -1.0);
        }
        if (e.opt) {
            apertures<LEAN>(r[k], e);
            exit_misalign<LEAN>(r[k], e);
        }
        if (!LEAN && (fl & ATB_F_SCALING)) change_pref<kFast>(r[k], e.f(ATB_SM_ISCALE));
    }
}

/* DriftPass.c:16-48 */
template <class T>
__device__ __forceinline__ void pass_drift(P6T<T>& r, RecipOf<T>& c, const Rec& e) {
    if (e.opt) {
        entrance_misalign(r, e);
        apertures(r, e);
    }
    drift6_pn<kFast>(r, e.f(ATB_DR_LE), opd_rcp(c, r.dp));
    if (e.opt) {
        apertures(r, e);
        exit_misalign(r, e);
    }
}

/* IdentityPass.c:20-43 */
template <class T>
__device__ __forceinline__ void pass_identity(P6T<T>& r, const Rec& e) {
    entrance_misalign(r, e);
    apertures(r, e);
    exit_misalign(r, e);
}

/* ThinMPolePass.c:28-70 */
template <class T>
__device__ __forceinline__ void pass_thinmpole(P6T<T>& r, const Rec& e, const Param& pm) {
    const uint32_t fl = e.flags();
    const int mo = e.mo();
    const double* A = e.p + ATB_TM_POLY;
    const double* B = A + mo + 1;
    Poly<-1> pl;
    pl.load(A, B, mo);
    if (pm.k >= 0) pl.set_param(pm.k, pm.v);
    const double bax = e.f(ATB_TM_BAX), bay = e.f(ATB_TM_BAY);
    if (fl & ATB_F_SCALING) change_pref<kFast>(r, e.f(ATB_TM_SCALE));
    entrance_misalign(r, e);
    apertures(r, e);
    strthinkick(r, pl, 1.0);
    r.px += bax * r.dp;
    r.py -= bay * r.dp;
    r.ct -= bax * r.x - bay * r.y;
    exit_misalign(r, e);
    if (fl & ATB_F_SCALING) change_pref<kFast>(r, e.f(ATB_TM_ISCALE));
}

/* RFCavityPass.c:23-68 -> attrackfunc.c:5-42 (trackRFCavity) */
template <class T>
__device__ __forceinline__ void rf_kick(P6T<T>& r, const Rec& e, int nturn) {
    const double nv = e.f(ATB_RF_NV), tf = e.f(ATB_RF_TF), lag = e.f(ATB_RF_LAG);
    const double ht = e.f(ATB_RF_HT), phi = e.f(ATB_RF_PHI);
    r.dp += -nv * sin(tf * ((r.ct - lag) / ATB_C0 - ht * (double)nturn) - phi);
}

template <class T>
__device__ __forceinline__ void pass_rfcavity(P6T<T>& r, const Rec& e, int nturn) {
    const uint32_t fl = e.flags();
    if (!(fl & ATB_F_THICK)) {
        if (fl & ATB_F_NV) rf_kick(r, e, nturn);
    } else {
        const double half = e.f(ATB_RF_HALF);
        drift6<kFast>(r, half);
        if (fl & ATB_F_NV) rf_kick(r, e, nturn);
        drift6<kFast>(r, half);
    }
}

/* CorrectorPass.c:25-90 */
template <class T>
__device__ __forceinline__ void pass_corrector(P6T<T>& r, const Rec& e) {
    const uint32_t fl = e.flags();
    const double xk = e.f(ATB_CO_XK), yk = e.f(ATB_CO_YK);
    if (fl & ATB_F_SCALING) change_pref<kFast>(r, e.f(ATB_CO_SCALE));
    if (!(fl & ATB_F_THICK)) {
        entrance_misalign(r, e);
        apertures(r, e);
        r.px += xk;
        r.py += yk;
    } else {
        const double le = e.f(ATB_CO_LE);
        T p_norm = 1.0 / (1.0 + r.dp);
        T nl = le * p_norm;
        entrance_misalign(r, e);
        apertures(r, e);
        r.ct += nl * p_norm * (e.f(ATB_CO_K2) + r.px * r.px + r.py * r.py + r.px * xk + r.py * yk) / 2;
        r.x += nl * (r.px + e.f(ATB_CO_HX));
        r.px += xk;
        r.y += nl * (r.py + e.f(ATB_CO_HY));
        r.py += yk;
        apertures(r, e);
    }
    exit_misalign(r, e);
    if (fl & ATB_F_SCALING) change_pref<kFast>(r, e.f(ATB_CO_ISCALE));
}

/* QuantDiffPass.c: random kicks keyed by (key, pbase + p, nturn, ei);
 * without a key (the derivative kernels) the element is the identity, as the
 * reference's envelope code disables it */
template <class T>
__device__ __forceinline__ void pass_quantdiff(P6T<T>& r, const Rec& e, const AtbRng* rng,
                                               long long p, int nturn, int ei) {
    if constexpr (!is_dual<T>::value) {
        if (rng) {
            double z[6];
            quantdiff_normals(rng->key, rng->pbase + p, nturn, ei, z);
            quantdiff_kick(r, e.p + ATB_QD_L, z);
        }
    }
}

template <class T>
__device__ __forceinline__ void track_element_any(P6T<T>& r, RecipOf<T>& c, const Rec& e,
                                                  int nturn, const Param& pm, const AtbRng* rng,
                                                  long long p, int ei) {
    switch (e.op()) {
        case ATB_OP_IDENTITY: pass_identity(r, e); break;
        case ATB_OP_DRIFT: pass_drift(r, c, e); break;
        case ATB_OP_STRMPOLE: pass_multipole_n<1, false, false>(&r, &c, e, pm); break;
        case ATB_OP_STRMPOLE_RAD: pass_multipole_n<1, false, true>(&r, &c, e, pm); break;
        case ATB_OP_BNDMPOLE: pass_multipole_n<1, true, false>(&r, &c, e, pm); break;
        case ATB_OP_BNDMPOLE_RAD: pass_multipole_n<1, true, true>(&r, &c, e, pm); break;
        case ATB_OP_THINMPOLE: pass_thinmpole(r, e, pm); break;
        case ATB_OP_RFCAVITY: pass_rfcavity(r, e, nturn); break;
        case ATB_OP_CORRECTOR: pass_corrector(r, e); break;
        case ATB_OP_APERTURE: check_rect(r, e.p + ATB_AP_LIM); break;
        case ATB_OP_QUANTDIFF: pass_quantdiff(r, e, rng, p, nturn, ei); break;
        default: break;
    }
}

/* the same out of line */
static __device__ __noinline__ P6 track_element_call(P6 r, Rec e, int nturn, Param pm,
                                                     const AtbRng* rng, long long p, int ei) {
    Recip c;
    track_element_any(r, c, e, nturn, pm, rng, p, ei);
    return r;
}

/* the field of a thin multipole, out of line: only x and y go there */
static __device__ __noinline__ double2 field_call(double x, double y, const double* A, int mo,
                                                  Param pm) {
    Poly<-1> pl;
    pl.load(A, A + mo + 1, mo);
    if (pm.k >= 0) pl.set_param(pm.k, pm.v);
    double2 f;
    pl.field(x, y, f.x, f.y);
    return f;
}

/* A magnet of a table compiled for another integrator of the GPU call, in the
 * kernels built with them (GEN); the hosts of the other kernels send them none
 * (atb_track_noalloc checks its raw table with a scan kernel, the tangent host
 * refuses it). */
__device__ __forceinline__ void track_integ(P6& r, Recip& c, const Rec& e, const Param& pm) {
    switch (e.op()) {
        case ATB_OP_STRMPOLE: pass_multipole_n<1, false, false, true>(&r, &c, e, pm); break;
        case ATB_OP_STRMPOLE_RAD: pass_multipole_n<1, false, true, true>(&r, &c, e, pm); break;
        case ATB_OP_BNDMPOLE: pass_multipole_n<1, true, false, true>(&r, &c, e, pm); break;
        default: pass_multipole_n<1, true, true, true>(&r, &c, e, pm); break;
    }
}

/* One element on one particle; lost particles (x is NaN) are skipped as every
 * reference pass method does (e.g. StrMPoleSymplectic4Pass.c:59).  Only what
 * most of a lattice consists of is in line: drifts, magnets (not with CALL),
 * markers, plain correctors, and of thin multipoles and apertures all but the
 * arithmetic on x and y.  With cavities, fringes and the rest beside them the
 * particle moved between registers around every element (159 instructions for
 * a drift, 14 of them FP64, where it now takes 88; a quadrupole beside its
 * steps 1,020 cycles of a lone warp instead of 1,400).  A call that takes and
 * returns the whole particle costs some 600 cycles: with it a marker took 1,400,
 * now 720, a thin multipole 2,000, now 1,200, a drift with apertures 2,300, now
 * 1,700. */
template <bool GEN = false, bool CALL = false, class T>
__device__ __forceinline__ void track_element(P6T<T>& r, RecipOf<T>& c, const Rec& e, int nturn,
                                              const Param& pm = Param{-1, 0.0},
                                              const AtbRng* rng = nullptr, long long p = 0,
                                              int ei = 0) {
    if (isnan(val(r.x))) return;
    if constexpr (is_dual<T>::value) {
        track_element_any(r, c, e, nturn, pm, rng, p, ei);
    } else {
        const int op = e.op();
        if (op == ATB_OP_DRIFT && e.opt == 0) {
            drift6_pn<kFast>(r, e.f(ATB_DR_LE), opd_rcp(c, r.dp));
            return;
        }
        if constexpr (GEN) {
            /* in line: out of line their coefficients, read on every kick, come
               through generic addresses, 3 to 9 % slower on full SMs */
            if (e.flags() & ATB_F_INTEG) {
                track_integ(r, c, e, pm);
                return;
            }
        }
        if (!CALL && !(e.flags() & (ATB_F_SCALING | ATB_F_FQ_IN | ATB_F_FQ_OUT))) {
            if (op == ATB_OP_STRMPOLE) {
                pass_multipole_n<1, false, false, false, true>(&r, &c, e, pm);
                return;
            }
            if (op == ATB_OP_STRMPOLE_RAD) {
                pass_multipole_n<1, false, true, false, true>(&r, &c, e, pm);
                return;
            }
            if (op == ATB_OP_BNDMPOLE) {
                pass_multipole_n<1, true, false, false, true>(&r, &c, e, pm);
                return;
            }
            if (op == ATB_OP_BNDMPOLE_RAD) {
                pass_multipole_n<1, true, true, false, true>(&r, &c, e, pm);
                return;
            }
        }
        if (op == ATB_OP_IDENTITY && e.opt == 0) return;
        if (op == ATB_OP_CORRECTOR && e.opt == 0 &&
            !(e.flags() & (ATB_F_SCALING | ATB_F_THICK))) {
            r.px += e.f(ATB_CO_XK);
            r.py += e.f(ATB_CO_YK);
            return;
        }
        if (__builtin_expect(op == ATB_OP_DRIFT && !(e.opt & ~ATB_OPT_APERTURES), 0)) {
            apertures<true>(r, e);
            drift6_pn<kFast>(r, e.f(ATB_DR_LE), opd_rcp(c, r.dp));
            apertures<true>(r, e);
            return;
        }
        if (__builtin_expect(op == ATB_OP_THINMPOLE && e.opt == 0 &&
                             !(e.flags() & ATB_F_SCALING), 0)) {
            const double2 f = field_call(r.x, r.y, e.p + ATB_TM_POLY, e.mo(), pm);
            const double bax = e.f(ATB_TM_BAX), bay = e.f(ATB_TM_BAY);
            r.px = msub(r.px, 1.0, f.x);
            r.py = madd(r.py, 1.0, f.y);
            r.px += bax * r.dp;
            r.py -= bay * r.dp;
            r.ct -= bax * r.x - bay * r.y;
            return;
        }
        r = track_element_call(r, e, nturn, pm, rng, p, ei);
    }
}

/* The particles of a thread go through a thick multipole together when none
 * of them is lost (a lost particle skips every element). */
template <int NP>
__device__ __forceinline__ bool track_together(const P6 (&r)[NP], const Rec& e) {
    const int op = e.op();
    if (op != ATB_OP_STRMPOLE && op != ATB_OP_STRMPOLE_RAD && op != ATB_OP_BNDMPOLE &&
        op != ATB_OP_BNDMPOLE_RAD)
        return false;
    bool all = true;
#pragma unroll
    for (int k = 0; k < NP; ++k) all &= !isnan(r[k].x);
    return all;
}

template <int NP>
__device__ __forceinline__ void pass_multipoles_together(P6 (&r)[NP], Recip (&c)[NP],
                                                         const Rec& e) {
    const Param none{-1, 0.0};
    switch (e.op()) {
        case ATB_OP_STRMPOLE: pass_multipole_n<NP, false, false>(r, c, e, none); break;
        case ATB_OP_STRMPOLE_RAD: pass_multipole_n<NP, false, true>(r, c, e, none); break;
        case ATB_OP_BNDMPOLE: pass_multipole_n<NP, true, false>(r, c, e, none); break;
        default: pass_multipole_n<NP, true, true>(r, c, e, none); break;
    }
}

/* pyat/at.c:123: lost if any coordinate is non-finite or |r_n| > 1, n < 5 */
template <class T>
__device__ __forceinline__ bool is_bad(const P6T<T>& r) {
    if constexpr (!is_dual<T>::value) {
        /* nearly always every |r_n| < 1 and ct is finite, which the exponents
           show without a floating-point compare */
        const uint32_t m = 0x7fffffffu;
        const uint32_t a = max(rn_hi(r.x) & m, rn_hi(r.px) & m);
        const uint32_t b = max(rn_hi(r.y) & m, rn_hi(r.py) & m);
        if (max(max(a, b), rn_hi(r.dp) & m) < 0x3ff00000u && rn_below(r.ct, 0x7ff00000u))
            return false;
    }
    return !all_finite(r) || fabs(val(r.x)) > 1.0 || fabs(val(r.px)) > 1.0 ||
           fabs(val(r.y)) > 1.0 || fabs(val(r.py)) > 1.0 || fabs(val(r.dp)) > 1.0;
}

__device__ __forceinline__ void load6(const double* src, P6& r) {
    const double2* s = reinterpret_cast<const double2*>(src);
    double2 a = s[0], b = s[1], c = s[2];
    r.x = a.x; r.px = a.y; r.y = b.x; r.py = b.y; r.dp = c.x; r.ct = c.y;
}

/* the same through L2 only: in the serving loop a tile's state may have been
   written by another SM's block since this SM last cached those lines */
__device__ __forceinline__ void load6_cg(const double* src, P6& r) {
    const double2* s = reinterpret_cast<const double2*>(src);
    double2 a = __ldcg(s), b = __ldcg(s + 1), c = __ldcg(s + 2);
    r.x = a.x; r.px = a.y; r.y = b.x; r.py = b.y; r.dp = c.x; r.ct = c.y;
}

__device__ __forceinline__ void store6(double* dst, const P6& r) {
    double2* d = reinterpret_cast<double2*>(dst);
    d[0] = make_double2(r.x, r.px);
    d[1] = make_double2(r.y, r.py);
    d[2] = make_double2(r.dp, r.ct);
}

/* segment index of the q-th segment visited by this launch */
__device__ __forceinline__ int seg_at(const AtbJob& J, long long q) {
    if (q < J.nseg_first) return J.seg_first0 + (int)q;
    return (int)((q - J.nseg_first) % J.nseg_turn);
}

/* ---------------- the kernel --------------------------------------------- */

/* The serving loop's claim (one thread per block).  New work first: the
 * next tile the host has published (taken by compare-and-swap on the counter
 * only while it is below `published`, so a block never holds a claim the host
 * has not published).  Then the continuation rings, class 0 first: a tile
 * that has run a chunk of its job's turns and waits for the next (an entry is
 * taken once its `seq` shows it written).  Without work the block sleeps between looks;
 * it leaves when the host sets `stop`, or after ATB_SERVE_IDLE_NS with
 * nothing claimed anywhere (no tile in flight that could still re-enqueue),
 * or after a hundred times that while tiles are in flight, and in any case
 * after two hundred times that in one claim.  Returns 1 with
 * the tile and the turns of its job already run, or 0 to leave. */
__device__ __forceinline__ int serve_claim(const AtbServeCtl* ctl, int* counter,
                                           const AtbTile* tiles, const AtbServeRing& ring,
                                           int* inflight, int* status, AtbTile* tile,
                                           int* turn_off) {
    uint64_t t0 = global_ns();
    const uint64_t entry = t0;
    while (true) {
        if (ctl->stop) return 0;
        /* a hard bound on the whole claim, whatever resets the idle clock:
           the block leaves and the host launches the kernel again while
           published or re-enqueued work waits */
        if (global_ns() - entry > 200ULL * ATB_SERVE_IDLE_NS) {
            atomicOr(status, ATB_STATUS_IDLE);
            return 0;
        }
        const int pub = ctl->published;
        const int c = atomicAdd(counter, 0);
        if (c < pub) {
            if (atomicCAS(counter, c, c + 1) == c) {
                atomicAdd(inflight, 1);
                __threadfence_system();          /* records read after the flag */
                const int4 tw = __ldcg(reinterpret_cast<const int4*>(tiles + c));
                *tile = *reinterpret_cast<const AtbTile*>(&tw);
                *turn_off = 0;
                return 1;
            }
            continue;                            /* another block took it */
        }
        /* continuations, the lowest class first; an entry reserved by a
           producer and not yet written, or lost to another block, sends the
           claim back to the top */
        bool again = false;
        for (int q = 0; q < ring.nring && !again; ++q) {
            const int h = atomicAdd(ring.head + q, 0);
            const int t = atomicAdd(ring.tail + q, 0);
            if (h >= t) continue;
            const AtbServeCont* e = ring.slots + (size_t)q * ring.cap + (h & (ring.cap - 1));
            if (__ldcg(&e->seq) == h + 1 && atomicCAS(ring.head + q, h, h + 1) == h) {
                atomicAdd(inflight, 1);
                __threadfence();
                const int4 tw = __ldcg(reinterpret_cast<const int4*>(&e->tile));
                *tile = *reinterpret_cast<const AtbTile*>(&tw);
                *turn_off = __ldcg(&e->turn_off);
                return 1;
            }
            again = true;
        }
        if (again) {
            t0 = global_ns();
            continue;
        }
        const bool busy = atomicAdd(inflight, 0) > 0;
        const uint64_t limit = busy ? 100ULL * ATB_SERVE_IDLE_NS : ATB_SERVE_IDLE_NS;
        if (global_ns() - t0 > limit) {
            atomicOr(status, ATB_STATUS_IDLE);
            return 0;
        }
        __nanosleep(4000);
    }
}

/* Put a tile that has run `turn_off` turns of its job back in the
 * continuation ring of class q.  Returns false if that ring is full. */
__device__ __forceinline__ bool serve_requeue(const AtbServeRing& ring, const AtbTile& tile,
                                              int turn_off, int q) {
    q = q < 0 ? 0 : (q >= ring.nring ? ring.nring - 1 : q);
    const int h = atomicAdd(ring.head + q, 0);
    const int t = atomicAdd(ring.tail + q, 0);
    if (t - h >= ring.cap - 64) return false;      /* leave room for racing producers */
    const int idx = atomicAdd(ring.tail + q, 1);
    AtbServeCont* e = ring.slots + (size_t)q * ring.cap + (idx & (ring.cap - 1));
    e->tile = tile;
    e->turn_off = turn_off;
    __threadfence();
    atomicExch(&e->seq, idx + 1);
    return true;
}

#if ATB_KERNELS

/* the loss map of one particle, written once (pyat/at.c:115-161) */
__device__ __forceinline__ void record_loss(const AtbJob& J, const P6& r, long long p, int nturn,
                                            int ei) {
    J.lturn[p] = (unsigned)nturn;
    J.lelem[p] = (unsigned)ei;
    store6(J.lcoord + 6 * p, r);
}

/* The persistent tile loop.  NP particles per thread: particle k of thread t
 * in a tile is tile.first + k * blockDim + t, so every k stays coalesced; the
 * element parameters read from shared memory serve all NP particles, whose
 * dependency chains interleave.
 *
 * Refill (NP = 1, a compaction scratch area and a job cursor given): a job
 * tracked over whole turns with no refpts snapshots and no per-turn
 * statistics hands out its particles through job_next[job] instead of fixed
 * tile ranges.  At the end of every turn a block retires the particles that
 * were lost or finished their turns (final state and loss flag stored), moves
 * the survivors to its lowest threads when that frees a warp, and takes
 * not-yet-started particles of the same job into its free lanes; each lane
 * counts its own turns (RF phase, loss turn and random kicks use the
 * particle's turn).  Blocks so stay full while their job has particles left
 * instead of running a few survivors for all remaining turns. */
template <int NP, bool GEN = false, bool SERVE = false>
__device__ __forceinline__ void track_tiles(const AtbJob* __restrict__ jobs,
                                            const AtbTile* __restrict__ tiles, int ntiles,
                                            int* __restrict__ tile_counter,
                                            unsigned long long* __restrict__ job_next,
                                            int* __restrict__ status, int smem_cap_words,
                                            double* __restrict__ scratch,
                                            AtbServeArgs sv = AtbServeArgs{}) {
    extern __shared__ __align__(128) double smem[];
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ int s_tile;
    /* serving: the claimed tile, the turns of its job already run, the job's
       full turn count, and whether the block keeps its tile for the next
       chunk (continuation ring full) */
    __shared__ AtbTile s_ctile;
    __shared__ int s_toff, s_full, s_self;
    __shared__ unsigned long long s_first;
    __shared__ int s_warp[ATB_MAX_THREADS / 32];
    double* buf0 = smem;
    double* buf1 = smem + smem_cap_words;
    uint32_t use_count[2] = {0u, 0u};
    const int tid = threadIdx.x;
    const int nthr = blockDim.x;

    if (tid == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_mbar_init();
    }
    if constexpr (SERVE) {
        if (tid == 0) s_self = 0;
    }
    __syncthreads();

    int resident_job = -1;   /* job whose whole table sits in buf0 */

    while (true) {
        if (tid == 0) {
            if constexpr (SERVE) {
                if (s_self) s_tile = 1;            /* the same tile, next chunk */
                else s_tile = serve_claim(sv.ctl, tile_counter, tiles, sv.ring, sv.inflight,
                                          status, &s_ctile, &s_toff);
            } else {
                s_tile = atomicAdd(tile_counter, 1);
            }
        }
        __syncthreads();
        const int t = s_tile;
        __syncthreads();
        if constexpr (SERVE) {
            if (t <= 0) break;
        } else {
            if (t >= ntiles) break;
        }
        AtbTile tile;
        const AtbJob* jp;
        if constexpr (SERVE) {
            /* the host writes job records while the kernel runs: read the
               record past the L1 cache into shared memory (only the serving
               kernel has this buffer), then narrow it to this claim's chunk
               of turns, continuing the absolute turn counter */
            __shared__ __align__(16) AtbJob s_job;
            tile = s_ctile;
            const unsigned long long* src =
                reinterpret_cast<const unsigned long long*>(jobs + tile.job);
            unsigned long long* dst = reinterpret_cast<unsigned long long*>(&s_job);
            for (int w = tid; w < (int)(sizeof(AtbJob) / 8); w += nthr) dst[w] = __ldcg(src + w);
            __syncthreads();
            if (tid == 0) {
                const int full = s_job.nturns;
                const int rem = full - s_toff;
                s_full = full;
                s_job.turn0 += s_toff;
                s_job.nturns = (s_job.chunk > 0 && s_job.chunk < rem) ? s_job.chunk : rem;
            }
            __syncthreads();
            jp = &s_job;
        } else {
            tile = tiles[t];
            jp = jobs + tile.job;
        }
        const AtbJob& J = *jp;
        const bool refill =
            NP == 1 && scratch != nullptr && job_next != nullptr && atb_job_refills(&J);
        long long first = tile.first;
        int count = tile.count;
        if (refill) {
            if (tid == 0) s_first = atomicAdd(&job_next[tile.job], (unsigned long long)count);
            __syncthreads();
            first = (long long)s_first;
            const long long left = J.np - first;
            if (left < count) count = left > 0 ? (int)left : 0;
            if (count == 0) continue;   /* the job's particles are all taken */
        }
        long long taken = count;        /* particles this claim stores (serving) */
        long long p[NP];
        bool active[NP];
        int lt0[NP];                    /* turn of the block at which the lane's particle joined */
        int tt_end = J.nturns;          /* the block tracks until this turn */
        bool exhausted = false;         /* the job cursor has no particle left */
        const bool resident = (J.resident != 0);

        /* read once: a store to global memory would have the element loop
           read them from the job again */
        const bool check_loss = J.check_loss != 0, losses = J.losses != 0;

        P6 r[NP];
        Recip rc[NP];
        bool lost[NP];
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            p[k] = first + (long long)k * nthr + tid;
            active[k] = (k * nthr + tid) < count;
            if constexpr (SERVE) {
                if (J.pidx && active[k]) p[k] = __ldcg(J.pidx + p[k]);
            }
            lt0[k] = 0;
            lost[k] = false;
            if (active[k]) {
                if constexpr (SERVE) {
                    load6_cg(J.r + 6 * p[k], r[k]);
                    if (J.losses) lost[k] = __ldcg(J.lost + p[k]) != 0;
                } else {
                    load6(J.r + 6 * p[k], r[k]);
                    if (J.losses) lost[k] = J.lost[p[k]] != 0;
                }
            } else {
                r[k].x = nan_d(); r[k].px = r[k].py = r[k].y = r[k].dp = r[k].ct = 0.0;
                lost[k] = true;
            }
        }

        /* staging pipeline state for this tile */
        /* segments the tile visits; a refilling block runs until its lanes
           are empty and leaves through the drain below */
        const long long nq = (J.nturns <= 0) ? 0
                             : refill ? (1LL << 60)
                                      : (long long)J.nseg_first +
                                            (long long)(J.nturns - 1) * J.nseg_turn;
        bool timed_out = false;
        if (resident) {
            if (resident_job != tile.job) {
                if (tid == 0) {
                    const uint32_t bytes = (uint32_t)(J.segs[0].nwords * 8);
                    mbar_expect_tx(&bars[0], bytes);
                    bulk_g2s(buf0, J.table + J.segs[0].word0, bytes, &bars[0]);
                }
                bool ok = mbar_wait_bounded(&bars[0], use_count[0] & 1u);
                use_count[0]++;
                timed_out = __syncthreads_or(!ok);
                resident_job = tile.job;
            }
        } else {
            resident_job = -1;
            if (tid == 0) {
                for (int b = 0; b < 2 && b < nq; ++b) {
                    const AtbSeg sg = J.segs[seg_at(J, b)];
                    const uint32_t bytes = (uint32_t)(sg.nwords * 8);
                    mbar_expect_tx(&bars[b], bytes);
                    bulk_g2s(b ? buf1 : buf0, J.table + sg.word0, bytes, &bars[b]);
                }
            }
        }
        if (timed_out) {
            if (tid == 0) atomicOr(status, ATB_STATUS_WAIT_TIMEOUT);
            break;
        }

        long long slot = J.rout_slot0;
        long long q = 0;
        for (int tt = 0; tt < tt_end && !timed_out; ++tt) {
            int nturn[NP];
#pragma unroll
            for (int k = 0; k < NP; ++k) nturn[k] = J.turn0 + tt - lt0[k];
            const int estart = (tt == 0) ? J.start_elem : 0;
            const int eend = J.end_elem;
            int nri = 0;
            unsigned nextref = (nri < J.nref) ? J.refpts[nri++] : 0xffffffffu;
            const int nseg_this = (tt == 0) ? J.nseg_first : J.nseg_turn;
            for (int si = 0; si < nseg_this; ++si, ++q) {
                const int b = resident ? 0 : (int)(q & 1);
                const AtbSeg sg = J.segs[resident ? 0 : seg_at(J, q)];
                const double* base = b ? buf1 : buf0;
                if (!resident) {
                    bool ok = mbar_wait_bounded(&bars[b], use_count[b] & 1u);
                    use_count[b]++;
                    if (__syncthreads_or(!ok)) { timed_out = true; break; }
                }
                /* elements of this segment */
                int e_lo = resident ? estart : sg.first_elem;
                int e_hi = resident ? eend : sg.first_elem + sg.nelem;
                if (e_lo < estart) e_lo = estart;
                if (e_hi > eend) e_hi = eend;
                int w = 0;
                if (resident) {
                    w = J.elem_off[e_lo] - J.elem_off[0];
                } else {
                    w = J.elem_off[e_lo] - J.elem_off[sg.first_elem];
                }
                for (int ei = e_lo; ei < e_hi; ++ei) {
                    Rec e;
                    e.p = base + w;
                    const uint64_t* hp = reinterpret_cast<const uint64_t*>(e.p);
                    e.hdr = hp[0];
                    e.opt = hp[1];
                    if ((unsigned)ei == nextref) {
#pragma unroll
                        for (int k = 0; k < NP; ++k)
                            if (active[k]) store6(J.rout + 6 * (p[k] + J.np * slot), r[k]);
                        ++slot;
                        nextref = (nri < J.nref) ? J.refpts[nri++] : 0xffffffffu;
                    }
                    bool together = false;
                    if constexpr (NP > 1) together = track_together(r, e);
                    if (together) {
                        if constexpr (NP > 1) pass_multipoles_together(r, rc, e);
                    } else {
#pragma unroll
                        for (int k = 0; k < NP; ++k)
                            track_element<GEN, (NP > 1)>(r[k], rc[k], e, nturn[k],
                                                         Param{-1, 0.0}, &J.rng, p[k], ei);
                    }
                    if (check_loss) {
#pragma unroll
                        for (int k = 0; k < NP; ++k) {
                            if (losses ? !lost[k] && is_bad(r[k])
                                       : isfinite(r[k].x) && is_bad(r[k])) {
                                if (losses && active[k])
                                    record_loss(J, r[k], p[k], nturn[k], ei);
                                lost[k] = true;
                                r[k].x = nan_d(); r[k].px = 0.0; r[k].y = 0.0;
                                r[k].py = 0.0; r[k].dp = 0.0; r[k].ct = 0.0;
                            }
                        }
                    }
                    w += e.len();
                }
                if (!resident) {
                    __syncthreads();   /* every thread is done with buffer b */
                    if (tid == 0 && q + 2 < nq) {
                        const AtbSeg nx = J.segs[seg_at(J, q + 2)];
                        const uint32_t bytes = (uint32_t)(nx.nwords * 8);
                        mbar_expect_tx(&bars[b], bytes);
                        bulk_g2s(b ? buf1 : buf0, J.table + nx.word0, bytes, &bars[b]);
                    }
                }
            }
            if (timed_out) break;
            if ((unsigned)J.nelem == nextref) {
#pragma unroll
                for (int k = 0; k < NP; ++k)
                    if (active[k]) store6(J.rout + 6 * (p[k] + J.np * slot), r[k]);
                ++slot;
            }
            if (J.alive) {
                /* per-turn survivors and first/second moments: warp ballot
                 * and shuffle reductions, one atomic per warp */
                unsigned cnt = 0;
                double v[12];
#pragma unroll
                for (int c = 0; c < 12; ++c) v[c] = 0.0;
#pragma unroll
                for (int k = 0; k < NP; ++k) {
                    const bool alive = active[k] && !isnan(r[k].x) && !(J.losses && lost[k]);
                    cnt += __popc(__ballot_sync(0xffffffffu, alive));
                    const double c6[6] = {r[k].x, r[k].px, r[k].y, r[k].py, r[k].dp, r[k].ct};
#pragma unroll
                    for (int c = 0; c < 6; ++c) {
                        const double x = alive ? c6[c] : 0.0;
                        v[c] += x;
                        v[6 + c] += x * x;
                    }
                }
#pragma unroll
                for (int c = 0; c < 12; ++c) {
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) v[c] += __shfl_xor_sync(0xffffffffu, v[c], o);
                }
                if ((tid & 31) == 0) {
                    atomicAdd(&J.alive[tt], cnt);
                    if (J.moments) {
#pragma unroll
                        for (int c = 0; c < 12; ++c) atomicAdd(&J.moments[12 * tt + c], v[c]);
                    }
                }
            }
            /* a tile whose particles are all lost stops early (nothing it
               would still compute is observable without refpts snapshots) */
            if (refill || (J.nref == 0 && tt + 1 < tt_end)) {
                if constexpr (NP == 1) {
                    if (refill && active[0]) {
                        /* retire a particle that is lost or has done its turns */
                        const bool done = tt + 1 - lt0[0] == J.nturns;
                        if (done || isnan(r[0].x) || (J.losses && lost[0])) {
                            store6(J.r + 6 * p[0], r[0]);
                            if (J.losses) J.lost[p[0]] = lost[0] ? 1 : 0;
                            active[0] = false;
                            r[0].x = nan_d(); r[0].px = 0.0; r[0].y = 0.0;
                            r[0].py = 0.0; r[0].dp = 0.0; r[0].ct = 0.0;
                            lost[0] = true;
                        }
                    }
                }
                bool any_live = false;
#pragma unroll
                for (int k = 0; k < NP; ++k)
                    any_live |= active[k] && !isnan(r[k].x) && !(J.losses && lost[k]);
                int nlive = __syncthreads_count(any_live);
                if constexpr (NP == 1) {
                    const bool live = any_live;
                    const unsigned ball = __ballot_sync(0xffffffffu, live);
                    const int lane = tid & 31, warp = tid >> 5;
                    /* warps that still hold a live particle */
                    const int held = __syncthreads_count(lane == 0 && ball != 0u);
                    if (scratch && nlive > 0 && (nlive + 31) / 32 < held) {
                        /* The survivors fit in fewer warps than hold them:
                           move them to the lowest threads, so that whole
                           warps fall idle instead of running with masked
                           lanes.  The lost ones are retired first (their
                           final state and loss flag are what the end of the
                           tile would store). */
                        if (active[0] && !live) {
                            store6(J.r + 6 * p[0], r[0]);
                            if (J.losses) J.lost[p[0]] = lost[0] ? 1 : 0;
                        }
                        if (lane == 0) s_warp[warp] = __popc(ball);
                        __syncthreads();
                        int dest = __popc(ball & ((1u << lane) - 1u));
                        for (int wv = 0; wv < warp; ++wv) dest += s_warp[wv];
                        double* sb = scratch + (size_t)blockIdx.x * ATB_COMPACT_WORDS * nthr;
                        if (live) {
                            sb[dest] = r[0].x;
                            sb[nthr + dest] = r[0].px;
                            sb[2 * nthr + dest] = r[0].y;
                            sb[3 * nthr + dest] = r[0].py;
                            sb[4 * nthr + dest] = r[0].dp;
                            sb[5 * nthr + dest] = r[0].ct;
                            sb[6 * nthr + dest] = __longlong_as_double(p[0]);
                            sb[7 * nthr + dest] = __longlong_as_double(lt0[0]);
                        }
                        __syncthreads();
                        active[0] = tid < nlive;
                        if (active[0]) {
                            r[0].x = sb[tid];
                            r[0].px = sb[nthr + tid];
                            r[0].y = sb[2 * nthr + tid];
                            r[0].py = sb[3 * nthr + tid];
                            r[0].dp = sb[4 * nthr + tid];
                            r[0].ct = sb[5 * nthr + tid];
                            p[0] = __double_as_longlong(sb[6 * nthr + tid]);
                            lt0[0] = (int)__double_as_longlong(sb[7 * nthr + tid]);
                            lost[0] = false;
                        } else {
                            r[0].x = nan_d(); r[0].px = 0.0; r[0].y = 0.0;
                            r[0].py = 0.0; r[0].dp = 0.0; r[0].ct = 0.0;
                            lost[0] = true;
                        }
                        __syncthreads();   /* scratch free for the next compaction */
                    }
                    if (refill && !exhausted) {
                        /* free lanes take the job's next particles */
                        const bool fr = !active[0];
                        const unsigned fb = __ballot_sync(0xffffffffu, fr);
                        if (lane == 0) s_warp[warp] = __popc(fb);
                        const int nfree = __syncthreads_count(fr);
                        if (nfree > 0) {
                            if (tid == 0)
                                s_first = atomicAdd(&job_next[tile.job],
                                                    (unsigned long long)nfree);
                            __syncthreads();
                            const long long c = (long long)s_first;
                            long long take = J.np - c;
                            if (take > nfree) take = nfree;
                            if (take < nfree) exhausted = true;
                            if (take > 0) {
                                int rank = __popc(fb & ((1u << lane) - 1u));
                                for (int wv = 0; wv < warp; ++wv) rank += s_warp[wv];
                                if (fr && rank < take) {
                                    p[0] = c + rank;
                                    active[0] = true;
                                    lt0[0] = tt + 1;
                                    load6(J.r + 6 * p[0], r[0]);
                                    lost[0] = J.losses ? J.lost[p[0]] != 0 : false;
                                }
                                nlive += (int)take;
                                taken += take;
                                if (tt + 1 + J.nturns > tt_end) tt_end = tt + 1 + J.nturns;
                            }
                            __syncthreads();   /* s_warp and s_first free again */
                        }
                    }
                }
                if (nlive == 0) {
                    if (!resident) {
                        /* wait for the copies this tile has in flight: after q
                           consumed segments, segments [0, min(nq, q + 2)) were
                           issued, buffer b holding the ones with index % 2 == b */
                        const long long issued = (q + 2 < nq) ? q + 2 : nq;
                        for (int b = 0; b < 2; ++b) {
                            long long pending = (issued - b + 1) / 2 - (q - b + 1) / 2;
                            for (; pending > 0; --pending) {
                                if (!mbar_wait_bounded(&bars[b], use_count[b] & 1u))
                                    timed_out = true;
                                use_count[b]++;
                            }
                        }
                        __syncthreads();
                    }
                    break;
                }
            }
        }
        if (timed_out) {
            /* drain our own copies still in flight before leaving */
            if (!resident) {
                const long long issued = (q + 2 < nq) ? q + 2 : nq;
                for (int b = 0; b < 2; ++b) {
                    if (use_count[b] < (uint32_t)((issued + 1 - b) / 2)) {
                        mbar_wait_bounded(&bars[b], use_count[b] & 1u);
                    }
                }
            }
            if (tid == 0) atomicOr(status, ATB_STATUS_WAIT_TIMEOUT);
            break;
        }
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            if (active[k]) {
                store6(J.r + 6 * p[k], r[k]);
                if (J.losses) J.lost[p[k]] = lost[k] ? 1 : 0;
            }
        }
        if constexpr (SERVE) {
            /* the chunk is stored and visible device-wide: a tile with live
               particles and turns left goes back to the continuation ring
               (or, if the ring is full, stays with this block); otherwise its
               particles count as done.  With a particle index (NP = 1) the
               tile keeps only its live particles, their indices packed at
               the front of its range, and the others count as done now. */
            __threadfence();
            bool live = false;
#pragma unroll
            for (int k = 0; k < NP; ++k)
                live |= active[k] && !isnan(r[k].x) && !(J.losses && lost[k]);
            const int nlive = __syncthreads_count(live);
            const bool more = nlive > 0 && s_toff + J.nturns < s_full;
            int keep_count = count;
            if (NP == 1 && J.pidx && more && nlive < count) {
                const unsigned ball = __ballot_sync(0xffffffffu, live);
                const int lane = tid & 31, warp = tid >> 5;
                if (lane == 0) s_warp[warp] = __popc(ball);
                __syncthreads();
                if (tid == 0) {
                    int acc = 0;
                    for (int w = 0; w < (nthr + 31) / 32; ++w) {
                        const int c = s_warp[w];
                        s_warp[w] = acc;
                        acc += c;
                    }
                }
                __syncthreads();
                if (live) {
                    const int rank = s_warp[warp] + __popc(ball & ((1u << lane) - 1u));
                    J.pidx[tile.first + rank] = (int32_t)p[0];
                }
                __threadfence();
                __syncthreads();
                keep_count = nlive;
            }
            if (tid == 0) {
                const int ran = s_toff + J.nturns;
                bool requeued = false, keep = false;
                if (more && !sv.ctl->stop) {
                    AtbTile nt = tile;
                    nt.count = keep_count;
                    /* class: decade of the tile's remaining time, so that
                       tiles near their end go first */
                    const double key = (double)(s_full - ran) * J.turn_cost;
                    const int q = key >= 1.0 ? (int)floor(log10(key)) : 0;
                    requeued = serve_requeue(sv.ring, nt, ran, q);
                    if (!requeued) {
                        atomicOr(status, ATB_STATUS_RING_FULL);
                        keep = true;
                        s_toff = ran;
                        s_ctile = nt;
                    }
                }
                if (requeued || keep) {
                    if (keep_count < taken)
                        atomicAdd(&sv.done[tile.job], (unsigned long long)(taken - keep_count));
                } else if (!more) {
                    atomicAdd(&sv.done[tile.job], (unsigned long long)taken);
                }
                if (!keep) atomicSub(sv.inflight, 1);
                s_self = keep ? 1 : 0;
            }
        }
        /* all threads must be past the last segment before the buffers are
           re-filled by the next tile */
        __syncthreads();
    }
}

#if ATB_KERNELS & ATB_KERNEL_BASE
extern "C" __global__ void __launch_bounds__(ATB_MAX_THREADS)
ATB_CAT(atb_track_kernel, ATB_KSUFFIX)(const AtbJob* __restrict__ jobs,
                                       const AtbTile* __restrict__ tiles, int ntiles,
                                       int* __restrict__ tile_counter,
                                       unsigned long long* __restrict__ job_next,
                                       int* __restrict__ status, int smem_cap_words,
                                       double* __restrict__ scratch) {
    track_tiles<1>(jobs, tiles, ntiles, tile_counter, job_next, status, smem_cap_words,
                   scratch);
}
#endif

#if ATB_KERNELS & ATB_KERNEL_GEN
/* with the other integrators of the GPU call (tables with ATB_F_INTEG) */
extern "C" __global__ void __launch_bounds__(ATB_MAX_THREADS)
ATB_CAT(ATB_CAT(atb_track_kernel, ATB_KSUFFIX), _gen)(const AtbJob* __restrict__ jobs,
                                                      const AtbTile* __restrict__ tiles,
                                                      int ntiles, int* __restrict__ tile_counter,
                                                      unsigned long long* __restrict__ job_next,
                                                      int* __restrict__ status,
                                                      int smem_cap_words,
                                                      double* __restrict__ scratch) {
    track_tiles<1, true>(jobs, tiles, ntiles, tile_counter, job_next, status, smem_cap_words,
                         scratch);
}
#endif

#if ATB_KERNELS & ATB_KERNEL_SERVE
/* The serving loop's persistent kernel: new tiles come from a queue the host
   appends to while it runs (AtbServeCtl), continuations from the device-side
   ring; `done[job]` counts the particles of each job that have run all their
   turns (or were lost) and are back in memory.  No lane refill: a tile keeps
   its particles from chunk to chunk. */
extern "C" __global__ void __launch_bounds__(ATB_MAX_THREADS)
ATB_CAT(atb_serve_kernel, ATB_KSUFFIX)(const AtbJob* __restrict__ jobs,
                                       const AtbTile* __restrict__ tiles, AtbServeArgs sv,
                                       int* __restrict__ tile_counter, int* __restrict__ status,
                                       int smem_cap_words, double* __restrict__ scratch) {
    track_tiles<1, false, true>(jobs, tiles, 0, tile_counter, nullptr, status, smem_cap_words,
                                scratch, sv);
}
#endif

#if ATB_KERNELS & ATB_KERNEL_NP2
/* two particles per thread (the autotuner's particles-per-thread choice) */
extern "C" __global__ void __launch_bounds__(ATB_MAX_THREADS)
ATB_CAT(ATB_CAT(atb_track_kernel, ATB_KSUFFIX), _np2)(const AtbJob* __restrict__ jobs,
                                                      const AtbTile* __restrict__ tiles,
                                                      int ntiles, int* __restrict__ tile_counter,
                                                      unsigned long long* __restrict__ job_next,
                                                      int* __restrict__ status,
                                                      int smem_cap_words,
                                                      double* __restrict__ scratch) {
    track_tiles<2>(jobs, tiles, ntiles, tile_counter, job_next, status, smem_cap_words,
                   scratch);
}
#endif

#endif  // ATB_KERNELS

}  // namespace atb

#endif  // ATB_TRACK_KERNEL_CUH
