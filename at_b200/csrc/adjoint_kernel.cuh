/*
 * The adjoint kernels: reverse-mode derivatives of multi-turn tracking.
 *
 * For a scalar function of the final coordinates, L = sum_p g_p . r_p(T),
 * one backward sweep gives dL/d r_p(0) for every particle and dL/dK_q for
 * every differentiated strength K_q = PolynomB[k_q] of an element, whatever
 * the number of strengths (the tangent kernel carries one derivative
 * direction per input instead).  This is the vector-Jacobian product that a
 * torch.autograd backward pass needs.
 *
 * Forward (atb_adjoint_forward_kernel): the particles are tracked with the
 * strengths substituted, by the same pass-method code as every other kernel
 * of this unit ("exact" arithmetic, so the values equal the exact tracking
 * kernel's), and the state entering every stride-th turn is stored.
 *
 * Backward (two launches per turn, last turn first): the forward kernel
 * tracks the turn again from its entry state, every element's entry state
 * going to a scratch array ([element][particle][6], coalesced) -- or the
 * forward pass stored every turn's (memory permitting); then
 * atb_adjoint_turn_kernel walks the elements backwards with
 * lambda <- J_e^T lambda, J_e the element's Jacobian at its stored entry
 * state, and at an element that carries K_q,
 * dL/dK_q += (d r_out / d K_q) . lambda_out, summed over the block's particles
 * in shared memory and added to the global sum once per block.
 *
 * Element adjoints:
 *  - DriftPass, IdentityPass, AperturePass, RFCavityPass, thin
 *    CorrectorPass, ThinMPolePass and the non-radiating StrMPole/BndMPole
 *    Symplectic4 passes (plain or bend-edge entrance/exit, misaligned or
 *    not): written out by hand.  A thick magnet is walked backwards from its
 *    exit state (the next element's entry state): every stage is undone on
 *    (x, px, y, py) -- a drift or kick is its own inverse but for the sign --
 *    and reversed at the coordinates so found: the fastdrift
 *    (driftkick.c:37-48), and the kick (driftkick.c:51-115) with the field
 *    derivative F'(z) of F(z) = sum (B_n + i A_n) z^n from a second Horner
 *    recursion and dF/dB_k = z^k for the strength.  In a magnet of a focusing
 *    phase above two radians, where the undone coordinates would lose digits,
 *    the steps' entry states are kept instead (adj_strong_magnet).
 *  - every other element (radiating magnets, quadrupole fringes, field
 *    scaling, thick correctors, bend edges of method 3): J_e from a
 *    forward-mode evaluation of the whole element on dual numbers (6
 *    directions, 7 when the element carries a strength), out of line so that
 *    its registers do not weigh on the common path.
 * A particle that is lost (NaN, or lost during the turn) gets a NaN
 * cotangent and adds nothing to the strengths' gradient.
 *
 * Bound by dependent FP64 latency at 3.5 warps a scheduler (65,536 particles).
 * A turn of the FODO ring with 128 strengths backwards: 5.0 ms with the step
 * entries recomputed into shared memory and every step run twice more; 2.3 ms
 * with the stages undone from the exit (0.8 of it the tracking), which needs
 * no store and keeps one stage's coordinates instead of seven.
 */
#ifndef ATB_ADJOINT_KERNEL_CUH
#define ATB_ADJOINT_KERNEL_CUH

#include "track_kernel.cuh"

namespace atb {

#ifndef ATB_ADJ_MIN_BLOCKS
#define ATB_ADJ_MIN_BLOCKS 4   /* 128 registers a thread: the dual-number
                                  fallback spills, the common path does not */
#endif

struct Lam6 {
    double v[6];
    double g;          /* the element's strength gradient contribution */
};

__device__ __forceinline__ Param adj_param(const AtbAdjoint& A, int ei) {
    Param pm{-1, 0.0};
    if (A.pelem) {
        const int q = A.pelem[ei];
        if (q >= 0) { pm.k = A.porder[q]; pm.v = A.pvalue[q]; }
    }
    return pm;
}

__device__ __forceinline__ Rec adj_rec(const AtbAdjoint& A, int ei) {
    Rec e;
    e.p = A.table + A.elem_off[ei];
    const uint64_t* hp = reinterpret_cast<const uint64_t*>(e.p);
    e.hdr = hp[0];
    e.opt = hp[1];
    return e;
}

/* ---- transposed linear maps --------------------------------------------- */

/* lambda <- R^T lambda for the misalignment rotation of mult_r */
__device__ __forceinline__ void adj_mult_r(double* lam, const double* m, bool dense) {
    if (dense) {
        double o[6];
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            double s = 0.0;
#pragma unroll
            for (int i = 0; i < 6; ++i) s = fma(m[i + 6 * j], lam[i], s);
            o[j] = s;
        }
#pragma unroll
        for (int j = 0; j < 6; ++j) lam[j] = o[j];
    } else {
        /* x' = m0 x + m1 y, px' = m2 px + m3 py, y' = m4 x + m5 y,
           py' = m6 px + m7 py */
        const double lx = lam[0], lpx = lam[1], ly = lam[2], lpy = lam[3];
        lam[0] = fma(m[0], lx, m[4] * ly);
        lam[2] = fma(m[1], lx, m[5] * ly);
        lam[1] = fma(m[2], lpx, m[6] * lpy);
        lam[3] = fma(m[3], lpx, m[7] * lpy);
    }
}

__device__ __forceinline__ void adj_exit_misalign(double* lam, const Rec& e) {
    if (const double* r2 = e.blk(ATB_OPT_R2)) adj_mult_r(lam, r2, e.flags() & ATB_F_R2_DENSE);
}

__device__ __forceinline__ void adj_entrance_misalign(double* lam, const Rec& e) {
    if (const double* r1 = e.blk(ATB_OPT_R1)) adj_mult_r(lam, r1, e.flags() & ATB_F_R1_DENSE);
}

/* ---- drift --------------------------------------------------------------- */

/* drift6 at input s: x += nl px, y += nl py, ct += nl pn S / 2 with
 * pn = 1/(1+dp), nl = L pn, S = px^2 + py^2 */
__device__ __forceinline__ void adj_drift6(const P6& s, double* lam, double L, double pn) {
    const double nl = L * pn;
    const double lx = lam[0], ly = lam[2], lc = lam[5];
    const double S = fma(s.px, s.px, s.py * s.py);
    const double cp = lc * nl * pn;
    lam[1] += fma(lx, nl, cp * s.px);
    lam[3] += fma(ly, nl, cp * s.py);
    lam[4] -= L * pn * pn * fma(lx, s.px, fma(ly, s.py, lc * pn * S));
}

/* DriftPass.c:16-48 */
__device__ __forceinline__ void adj_pass_drift(const P6& s, Recip& rc, double* lam,
                                               const Rec& e) {
    if (!e.opt) {
        adj_drift6(s, lam, e.f(ATB_DR_LE), opd_rcp(rc, s.dp));
        return;
    }
    P6 r = s;
    entrance_misalign(r, e);
    adj_exit_misalign(lam, e);
    adj_drift6(r, lam, e.f(ATB_DR_LE), opd_rcp(rc, r.dp));
    adj_entrance_misalign(lam, e);
}

/* ---- thick multipoles ---------------------------------------------------- */

/* The element's multipole coefficients for the reverse pass, B_sk replaced
 * by the differentiated strength kv: in registers for MaxOrder MO in 0..3
 * (SKEW false: every A_n is zero), read from the table for MO = -1 (any
 * order).  field() is F(z) = sum_n (B_n + i A_n) z^n by Horner's rule with
 * fused multiply-adds (the recomputed steps inside an element only feed
 * derivatives, so they need not round as the tracking does); prime() is F'(z)
 * by the same recursion. */
template <int MO, bool SKEW>
struct AdjCoef {
    double a[SKEW ? MO + 1 : 1], b[MO + 1];
    int sk;
    __device__ __forceinline__ void load(const double* A, const double* B, int, int k,
                                         double v) {
#pragma unroll
        for (int i = 0; i <= MO; ++i) {
            if (SKEW) a[SKEW ? i : 0] = A[i];
            b[i] = (i == k) ? v : B[i];
        }
        sk = k;
    }
    __device__ __forceinline__ double an(int i) const { return SKEW ? a[SKEW ? i : 0] : 0.0; }
    __device__ __forceinline__ void field(double x, double y, double& re, double& im) const {
        if constexpr (SKEW || MO == 0) {
            re = b[MO];
            im = an(MO);
#pragma unroll
            for (int i = MO - 1; i >= 0; --i) {
                const double t = fma(re, x, fma(-im, y, b[i]));
                im = fma(im, x, fma(re, y, an(i)));
                re = t;
            }
        } else {
            re = fma(b[MO], x, b[MO - 1]);
            im = b[MO] * y;
#pragma unroll
            for (int i = MO - 2; i >= 0; --i) {
                const double t = fma(re, x, fma(-im, y, b[i]));
                im = fma(im, x, re * y);
                re = t;
            }
        }
    }
    __device__ __forceinline__ void prime(double x, double y, double& dr, double& di) const {
        if constexpr (MO == 0) {
            dr = 0.0;
            di = 0.0;
        } else if constexpr (!SKEW && MO == 1) {
            dr = b[1];
            di = 0.0;
        } else if constexpr (!SKEW) {
            dr = fma((double)MO * b[MO], x, (double)(MO - 1) * b[MO - 1]);
            di = (double)MO * b[MO] * y;
#pragma unroll
            for (int n = MO - 2; n >= 1; --n) {
                const double t = fma(dr, x, fma(-di, y, (double)n * b[n]));
                di = fma(di, x, dr * y);
                dr = t;
            }
        } else {
            dr = (double)MO * b[MO];
            di = (double)MO * an(MO);
#pragma unroll
            for (int n = MO - 1; n >= 1; --n) {
                const double t = fma(dr, x, fma(-di, y, (double)n * b[n]));
                di = fma(di, x, fma(dr, y, (double)n * an(n)));
                dr = t;
            }
        }
    }
};

template <>
struct AdjCoef<-1, true> {
    const double* a;
    const double* b;
    int mo;
    int sk;
    double kv;
    __device__ __forceinline__ void load(const double* A, const double* B, int m, int k,
                                         double v) {
        a = A; b = B; mo = m; sk = k; kv = v;
    }
    __device__ __forceinline__ double bk(int i) const { return (i == sk) ? kv : b[i]; }
    __device__ __forceinline__ void field(double x, double y, double& re, double& im) const {
        re = bk(mo);
        im = a[mo];
        for (int i = mo - 1; i >= 0; --i) {
            const double t = fma(re, x, fma(-im, y, bk(i)));
            im = fma(im, x, fma(re, y, a[i]));
            re = t;
        }
    }
    __device__ __forceinline__ void prime(double x, double y, double& dr, double& di) const {
        if (mo <= 0) {
            dr = 0.0;
            di = 0.0;
            return;
        }
        dr = (double)mo * bk(mo);
        di = (double)mo * a[mo];
        for (int n = mo - 1; n >= 1; --n) {
            const double t = fma(dr, x, fma(-di, y, (double)n * bk(n)));
            di = fma(di, x, fma(dr, y, (double)n * a[n]));
            dr = t;
        }
    }
};

/* (x + i y)^k */
__device__ __forceinline__ void zpow(double x, double y, int k, double& zr, double& zi) {
    zr = 1.0;
    zi = 0.0;
    for (int i = 0; i < k; ++i) {
        const double t = fma(zr, x, -zi * y);
        zi = fma(zr, y, zi * x);
        zr = t;
    }
}

/* strthinkick / bndthinkick of length L at input (x, y):
 * px -= L (Re F - [bend] (dp - x irho) irho), py += L Im F,
 * [bend] ct += lirho x */
template <bool BEND, class C>
__device__ __forceinline__ void adj_kick(const C& c, double x, double y, double L, double lirho,
                                         double irho, double* lam, double& g) {
    double dr, di;
    c.prime(x, y, dr, di);
    const double lpx = lam[1], lpy = lam[3];
    const double ay = L * dr, b = L * di;
    if (BEND) {
        const double li = L * irho;
        lam[0] = fma(-fma(li, irho, ay), lpx, fma(lirho, lam[5], lam[0]));
        lam[4] = fma(li, lpx, lam[4]);
    } else {
        lam[0] = fma(-ay, lpx, lam[0]);
    }
    lam[0] = fma(b, lpy, lam[0]);
    lam[2] = fma(ay, lpy, fma(b, lpx, lam[2]));
    if (c.sk >= 0) {
        double zr, zi;
        zpow(x, y, c.sk, zr, zi);
        g = fma(L, fma(-zr, lpx, zi * lpy), g);
    }
}

/* the same in an upright magnet up to the quadrupole, where F' = b1 */
template <bool BEND, int MO>
__device__ __forceinline__ void adj_kick(const AdjCoef<MO, false>& c, double x, double y, double L,
                                         double lirho, double irho, double* lam, double& g) {
    if constexpr (MO == 1) {
        const double lpx = lam[1], lpy = lam[3];
        const double ay = L * c.b[1];
        if (BEND) {
            const double li = L * irho;
            lam[0] = fma(-fma(li, irho, ay), lpx, fma(lirho, lam[5], lam[0]));
            lam[4] = fma(li, lpx, lam[4]);
        } else {
            lam[0] = fma(-ay, lpx, lam[0]);
        }
        lam[2] = fma(ay, lpy, lam[2]);
        if (c.sk >= 0) g = fma(L, fma(-x, lpx, y * lpy), g);     /* B_1, the only one */
    } else {
        adj_kick<BEND, AdjCoef<MO, false>>(c, x, y, L, lirho, irho, lam, g);
    }
}

/* fastdrift (exact form) at input (px, py): x += nl px, y += nl py,
 * ct += nl S h with h = 1/(2 (1 + dp)) and nl = L/(1 + dp_entry).  lam[5] is
 * the same all through a magnet, so c2 = 2 h nl lam[5] comes from outside, and
 * the momentum's share is left as two sums over the drifts of one length,
 * a = sum lx px + ly py and b = sum S (adj_drift_sums). */
struct DriftSums {
    double a, b;
};
__device__ __forceinline__ void adj_fastdrift(double px, double py, double nl, double c2,
                                              double* lam, DriftSums& d) {
    const double lx = lam[0], ly = lam[2];
    lam[1] = fma(lx, nl, fma(c2, px, lam[1]));
    lam[3] = fma(ly, nl, fma(c2, py, lam[3]));
    d.a = fma(lx, px, fma(ly, py, d.a));
    d.b = fma(px, px, fma(py, py, d.b));
}
/* what drifts of length nl add to the cotangent of the body's momentum (from
 * h), and to that of the entry's (from nl, times -1/(1 + dp_entry)) */
__device__ __forceinline__ void adj_drift_sums(const DriftSums& d, double nl, double h, double lc,
                                               double* lam, double& lnl) {
    const double t = lc * h * d.b;
    lam[4] = fma(-2.0 * nl * h, t, lam[4]);
    lnl = fma(nl, d.a + t, lnl);
}

/* The transverse coordinates inside a non-radiating magnet, where dp is
 * constant and ct feeds nothing: what the undone stages carry.  They feed
 * derivatives only and may differ from the tracked ones by roundings. */
struct XY {
    double x, px, y, py;
};

__device__ __forceinline__ void xy_drift(XY& q, double nl) {
    q.x = fma(nl, q.px, q.x);
    q.y = fma(nl, q.py, q.y);
}

/* a kick of length L; with -L, the kick undone */
template <bool BEND, class C>
__device__ __forceinline__ void xy_kick(XY& q, const C& c, double L, double irho, double dp) {
    double re, im;
    c.field(q.x, q.y, re, im);
    if (BEND) re = fma(-fma(-q.x, irho, dp), irho, re);     /* re - (dp - x irho) irho */
    q.px = fma(-L, re, q.px);
    q.py = fma(L, im, q.py);
}

/* edge_fringe (methods other than 3) at input (y, dp):
 * px += x fx, py -= y fy(dp) with fy = tn or tn/(1+dp) (method 2),
 * tn = irho tan(edge - fc/(1+dp)) (fy_c when that argument is the edge) */
__device__ __noinline__ double2 adj_edge_fringed(double dp, double irho, double edge, double fc,
                                                 double fy_c, int method, bool fc0) {
    const double opd = 1.0 + dp;
    double fy = fy_c, dfy = 0.0;
    if (!fc0) {
        const double t = edge - fc / opd;
        const double tt = tan(t);
        if (t != edge) fy = irho * tt;
        dfy = irho * fma(tt, tt, 1.0) * fc / (opd * opd);
    }
    if (method == ATB_BM_2) {
        fy = fy / opd;
        dfy = (dfy - fy) / opd;
    }
    return make_double2(fy, dfy);
}
__device__ __forceinline__ void adj_edge(double y, double dp, double* lam, double irho,
                                         const Rec& e, int w_edge, int method, bool fc0) {
    const double fy_c = e.f(w_edge + 3);
    double2 f = make_double2(fy_c, 0.0);
    if (!fc0 || method == ATB_BM_2)
        f = adj_edge_fringed(dp, irho, e.f(w_edge), e.f(w_edge + 1), fy_c, method, fc0);
    lam[0] = fma(lam[1], e.f(w_edge + 2), lam[0]);
    lam[4] = fma(-lam[3] * y, f.y, lam[4]);
    lam[2] = fma(-lam[3], f.x, lam[2]);
}

__device__ __forceinline__ double adj_edge_fy(double dp, double irho, const Rec& e, int w_edge,
                                              int method, bool fc0) {
    const double fy_c = e.f(w_edge + 3);
    if (fc0 && method != ATB_BM_2) return fy_c;
    return adj_edge_fringed(dp, irho, e.f(w_edge), e.f(w_edge + 1), fy_c, method, fc0).x;
}

/* the hand-written magnet path applies (flags and edge methods) */
__device__ __forceinline__ bool adj_by_hand(const Rec& e, bool bend) {
    const uint32_t fl = e.flags();
    if (fl & (ATB_F_SCALING | ATB_F_FQ_IN | ATB_F_FQ_OUT | ATB_F_INTEG)) return false;
    if (bend) {
        const int m_in = (int)((fl >> ATB_F_BM_IN_SHIFT) & ATB_F_BM_MASK);
        const int m_out = (int)((fl >> ATB_F_BM_OUT_SHIFT) & ATB_F_BM_MASK);
        if (m_in == ATB_BM_3 || m_out == ATB_BM_3) return false;
    }
    return true;
}

/* Undoing a stage rounds its coordinates, and the roundings grow by the inverse
 * of the magnet's map as the walk goes on: relative to the coordinates by about
 * exp(2 phi), phi^2 = |F'| L^2 the magnet's (worst) focusing phase.  Up to phi
 * = 2 dL/d r is as close to the tangent's as with forward coordinates (2e-15 of
 * its terms); the delta column is off by 6e-15 at phi = 3 and 2e-12 at 6.
 * Quadrupoles of the FODO and large ring have 0.5 and 0.6.  Stronger magnets,
 * at this particle's ends of it, keep their step entries (adj_strong_magnet).
 * k, nl: the magnet's kick and drift lengths. */
template <class C>
__device__ __forceinline__ bool adj_strong(const C& c, const XY& in, const XY& out, double k,
                                           double nl, double irho) {
    double ar, ai, br, bi;
    c.prime(in.x, in.y, ar, ai);
    c.prime(out.x, out.y, br, bi);
    const double f = fmax(fabs(ar) + fabs(ai), fabs(br) + fabs(bi));
    return fma(irho, irho, f) * fabs(k * nl) > 4.0;
}

/* A magnet in reverse with every coordinate found forwards: the transverse
 * coordinates entering its steps are kept (all of up to ten, every
 * ceil(n / 10)-th of more, the others tracked again from the nearest), each
 * step is run again with the inputs of its stages kept, and the stages are
 * reversed.  Twice the work of undoing them. */
template <bool BEND>
__device__ __noinline__ Lam6 adj_strong_magnet(P6 s, Lam6 io, Rec e, Param pm) {
    constexpr int KEEP = 10;
    double* lam = io.v;
    const uint32_t fl = e.flags();
    const double K1 = e.f(ATB_SM_K1), K2 = e.f(ATB_SM_K2);
    const int mo = e.mo(), ns = e.nsteps();
    const double* A = e.p + (BEND ? ATB_BM_POLY : ATB_SM_POLY);
    AdjCoef<-1, true> c;
    c.load(A, A + mo + 1, mo, pm.k, pm.v);
    const double pn0 = 1.0 / (1.0 + s.dp);
    const double nl1 = e.f(ATB_SM_L1) * pn0, nl2 = e.f(ATB_SM_L2) * pn0;
    const double irho = BEND ? e.f(ATB_BM_IRHO) : 0.0;
    const double k1i = BEND ? e.f(ATB_BM_K1IRHO) : 0.0, k2i = BEND ? e.f(ATB_BM_K2IRHO) : 0.0;
    const int m_in = (int)((fl >> ATB_F_BM_IN_SHIFT) & ATB_F_BM_MASK);
    const int m_out = (int)((fl >> ATB_F_BM_OUT_SHIFT) & ATB_F_BM_MASK);
    P6 r = s;
    entrance_misalign(r, e);
    const double dp = r.dp;
    XY q{r.x, r.px, r.y, r.py};
    if (BEND) {
        q.px = fma(q.x, e.f(ATB_BM_FXIN), q.px);
        q.py = fma(-q.y, adj_edge_fy(dp, irho, e, ATB_BM_EIN, m_in, fl & ATB_F_FC0_IN), q.py);
    }
    auto step = [&](XY& t) {
        xy_drift(t, nl1);
        xy_kick<BEND>(t, c, K1, irho, dp);
        xy_drift(t, nl2);
        xy_kick<BEND>(t, c, K2, irho, dp);
        xy_drift(t, nl2);
        xy_kick<BEND>(t, c, K1, irho, dp);
        xy_drift(t, nl1);
    };
    XY keep[KEEP];
    const int stride = ns > KEEP ? (ns + KEEP - 1) / KEEP : 1;
    for (int m = 0; m < ns; ++m) {
        if (m % stride == 0) keep[m / stride] = q;
        step(q);
    }
    adj_exit_misalign(lam, e);
    const double h = 0.5 / (1.0 + dp), lc = lam[5], cc = 2.0 * h * lc;
    const double c1 = cc * nl1, c2 = cc * nl2;
    if (BEND) adj_edge(q.y, dp, lam, irho, e, ATB_BM_EOUT, m_out, fl & ATB_F_FC0_OUT);
    DriftSums d1{0.0, 0.0}, d2{0.0, 0.0};
    for (int m = ns - 1; m >= 0; --m) {
        XY t = keep[m / stride];
        for (int j = (m / stride) * stride; j < m; ++j) step(t);
        const XY t0 = t;
        xy_drift(t, nl1);
        const XY t1 = t;
        xy_kick<BEND>(t, c, K1, irho, dp);
        xy_drift(t, nl2);
        const XY t3 = t;
        xy_kick<BEND>(t, c, K2, irho, dp);
        xy_drift(t, nl2);
        const XY t5 = t;
        xy_kick<BEND>(t, c, K1, irho, dp);
        adj_fastdrift(t.px, t.py, nl1, c1, lam, d1);
        adj_kick<BEND>(c, t5.x, t5.y, K1, k1i, irho, lam, io.g);
        adj_fastdrift(t5.px, t5.py, nl2, c2, lam, d2);
        adj_kick<BEND>(c, t3.x, t3.y, K2, k2i, irho, lam, io.g);
        adj_fastdrift(t3.px, t3.py, nl2, c2, lam, d2);
        adj_kick<BEND>(c, t1.x, t1.y, K1, k1i, irho, lam, io.g);
        adj_fastdrift(t0.px, t0.py, nl1, c1, lam, d1);
    }
    double lnl = 0.0;
    adj_drift_sums(d1, nl1, h, lc, lam, lnl);
    adj_drift_sums(d2, nl2, h, lc, lam, lnl);
    if (BEND) adj_edge(r.y, dp, lam, irho, e, ATB_BM_EIN, m_in, fl & ATB_F_FC0_IN);
    adj_entrance_misalign(lam, e);
    lam[4] = fma(-lnl, pn0, lam[4]);
    return io;
}

/* StrMPoleSymplectic4Pass.c:29-109 / BndMPoleSymplectic4Pass.c:38-129 in
 * reverse, from the entry state s and the exit state sx.  A magnet with
 * misalignments or apertures of its own finds the body's exit by tracking the
 * body again (undoing a rotation would need its inverse).  False: the magnet is
 * a strong one, nothing done. */
template <bool BEND, int MO, bool SKEW, bool PLAIN = false>
__device__ __forceinline__ bool adj_multipole_mo(const P6& s, const P6& sx, Recip& rc,
                                                 double* lam, const Rec& e, const Param& pm,
                                                 double& g) {
    const uint32_t fl = e.flags();
    const double K1 = e.f(ATB_SM_K1), K2 = e.f(ATB_SM_K2);
    const int mo = e.mo(), ns = e.nsteps();
    const double* A = e.p + (BEND ? ATB_BM_POLY : ATB_SM_POLY);
    AdjCoef<MO, SKEW> c;
    c.load(A, A + mo + 1, mo, pm.k, pm.v);
    const double pn0 = opd_rcp(rc, s.dp);
    const double nl1 = e.f(ATB_SM_L1) * pn0, nl2 = e.f(ATB_SM_L2) * pn0, nl11 = 2.0 * nl1;
    const double irho = BEND ? e.f(ATB_BM_IRHO) : 0.0;
    const double k1i = BEND ? e.f(ATB_BM_K1IRHO) : 0.0, k2i = BEND ? e.f(ATB_BM_K2IRHO) : 0.0;
    const int m_in = (int)((fl >> ATB_F_BM_IN_SHIFT) & ATB_F_BM_MASK);
    const int m_out = (int)((fl >> ATB_F_BM_OUT_SHIFT) & ATB_F_BM_MASK);

    /* q: leaving the body, before the exit edge */
    XY q{sx.x, sx.px, sx.y, sx.py}, q0{s.x, s.px, s.y, s.py};
    double dp = sx.dp;                       /* constant through the magnet */
    if (!PLAIN && e.opt) {
        P6 r = s;
        entrance_misalign(r, e);
        dp = r.dp;
        q = q0 = XY{r.x, r.px, r.y, r.py};
        if (BEND) {
            q.px = fma(q.x, e.f(ATB_BM_FXIN), q.px);
            q.py = fma(-q.y, adj_edge_fy(dp, irho, e, ATB_BM_EIN, m_in, fl & ATB_F_FC0_IN), q.py);
        }
#pragma unroll 1
        for (int i = 0; i < 3 * ns; ++i) {
            const bool mid = i % 3 == 1;
            xy_drift(q, i % 3 ? nl2 : i ? nl11 : nl1);
            xy_kick<BEND>(q, c, mid ? K2 : K1, irho, dp);
        }
        if (ns > 0) xy_drift(q, nl1);
    }
    if (adj_strong(c, q0, q, fma(2.0, K1, K2) * ns, 2.0 * (nl1 + nl2) * ns, irho)) return false;
    if (!PLAIN && e.opt) {
        adj_exit_misalign(lam, e);
    } else if (BEND) {
        q.px = fma(-q.x, e.f(ATB_BM_FXOUT), q.px);
        q.py = fma(q.y, adj_edge_fy(dp, irho, e, ATB_BM_EOUT, m_out, fl & ATB_F_FC0_OUT), q.py);
    }
    const double h = 0.5 * (PLAIN || dp == s.dp ? pn0 : 1.0 / (1.0 + dp));
    if (BEND) adj_edge(q.y, dp, lam, irho, e, ATB_BM_EOUT, m_out, fl & ATB_F_FC0_OUT);
    double lnl = 0.0;
    if (ns > 0) {
        const double lc = lam[5], cc = 2.0 * h * lc;
        const double c1 = cc * nl1, c2 = cc * nl2, c11 = cc * nl11;
        DriftSums d1{0.0, 0.0}, d11{0.0, 0.0}, d2{0.0, 0.0};
        adj_fastdrift(q.px, q.py, nl1, c1, lam, d1);
        xy_drift(q, -nl1);
        for (int m = ns;;) {
            adj_kick<BEND>(c, q.x, q.y, K1, k1i, irho, lam, g);
            xy_kick<BEND>(q, c, -K1, irho, dp);
            adj_fastdrift(q.px, q.py, nl2, c2, lam, d2);
            xy_drift(q, -nl2);
            adj_kick<BEND>(c, q.x, q.y, K2, k2i, irho, lam, g);
            xy_kick<BEND>(q, c, -K2, irho, dp);
            adj_fastdrift(q.px, q.py, nl2, c2, lam, d2);
            xy_drift(q, -nl2);
            adj_kick<BEND>(c, q.x, q.y, K1, k1i, irho, lam, g);
            xy_kick<BEND>(q, c, -K1, irho, dp);
            if (--m == 0) break;
            /* a step's first drift and the last of the step before it */
            adj_fastdrift(q.px, q.py, nl11, c11, lam, d11);
            xy_drift(q, -nl11);
        }
        adj_fastdrift(q.px, q.py, nl1, c1, lam, d1);
        xy_drift(q, -nl1);
        adj_drift_sums(d1, nl1, h, lc, lam, lnl);
        adj_drift_sums(d11, nl11, h, lc, lam, lnl);
        adj_drift_sums(d2, nl2, h, lc, lam, lnl);
    }
    if (BEND) adj_edge(q.y, dp, lam, irho, e, ATB_BM_EIN, m_in, fl & ATB_F_FC0_IN);
    if (!PLAIN && e.opt) adj_entrance_misalign(lam, e);
    /* nl = L / (1 + dp) of the entry momentum */
    lam[4] = fma(-lnl, pn0, lam[4]);
    return true;
}

template <bool BEND>
__device__ __forceinline__ void adj_pass_multipole(const P6& s, const P6& sx, Recip& rc,
                                                   double* lam, const Rec& e, const Param& pm,
                                                   double& g) {
    const bool upright = e.flags() & ATB_F_NOSKEW;
    const int mo = e.mo();
    bool done;
    if (mo == 1 && upright) done = adj_multipole_mo<BEND, 1, false>(s, sx, rc, lam, e, pm, g);
    else if (mo == 2 && upright) done = adj_multipole_mo<BEND, 2, false>(s, sx, rc, lam, e, pm, g);
    else if (mo == 3 && upright) done = adj_multipole_mo<BEND, 3, false>(s, sx, rc, lam, e, pm, g);
    else if (mo == 0) done = adj_multipole_mo<BEND, 0, true>(s, sx, rc, lam, e, pm, g);
    else done = adj_multipole_mo<BEND, -1, true>(s, sx, rc, lam, e, pm, g);
    if (done) return;
    Lam6 io;
#pragma unroll
    for (int i = 0; i < 6; ++i) io.v[i] = lam[i];
    io.g = g;
    io = adj_strong_magnet<BEND>(s, io, e, pm);
#pragma unroll
    for (int i = 0; i < 6; ++i) lam[i] = io.v[i];
    g = io.g;
}

/* ---- thin elements -------------------------------------------------------- */

/* rf_kick at input s: dp -= nv sin(tf ((ct - lag)/c - ht nturn) - phi) */
__device__ __forceinline__ void adj_rf_kick(const P6& s, double* lam, const Rec& e, int nturn) {
    const double nv = e.f(ATB_RF_NV), tf = e.f(ATB_RF_TF), lag = e.f(ATB_RF_LAG);
    const double ht = e.f(ATB_RF_HT), phi = e.f(ATB_RF_PHI);
    const double a = tf * ((s.ct - lag) / ATB_C0 - ht * (double)nturn) - phi;
    lam[5] = fma(-nv * cos(a) * tf / ATB_C0, lam[4], lam[5]);
}

/* RFCavityPass.c:23-68 (trackRFCavity, attrackfunc.c:5-42) */
__device__ __forceinline__ void adj_pass_rfcavity(const P6& s, double* lam, const Rec& e,
                                                  int nturn) {
    const uint32_t fl = e.flags();
    if (!(fl & ATB_F_THICK)) {
        if (fl & ATB_F_NV) adj_rf_kick(s, lam, e, nturn);
        return;
    }
    const double half = e.f(ATB_RF_HALF);
    P6 r = s;
    drift6<false>(r, half);
    const P6 s1 = r;
    if (fl & ATB_F_NV) rf_kick(r, e, nturn);
    adj_drift6(r, lam, half, 1.0 / (1.0 + r.dp));
    if (fl & ATB_F_NV) adj_rf_kick(s1, lam, e, nturn);
    adj_drift6(s, lam, half, 1.0 / (1.0 + s.dp));
}

/* ThinMPolePass.c:28-70 without field scaling */
__device__ __forceinline__ void adj_pass_thinmpole(const P6& s, double* lam, const Rec& e,
                                                   const Param& pm, double& g) {
    const int mo = e.mo();
    const double* A = e.p + ATB_TM_POLY;
    const double* B = A + mo + 1;
    const double bax = e.f(ATB_TM_BAX), bay = e.f(ATB_TM_BAY);
    P6 r = s;
    entrance_misalign(r, e);
    adj_exit_misalign(lam, e);
    /* px += bax dp, py -= bay dp, ct -= bax x - bay y */
    lam[4] = fma(bax, lam[1], fma(-bay, lam[3], lam[4]));
    lam[0] = fma(-bax, lam[5], lam[0]);
    lam[2] = fma(bay, lam[5], lam[2]);
    AdjCoef<-1, true> c;
    c.load(A, B, mo, pm.k, pm.v);
    adj_kick<false>(c, r.x, r.y, 1.0, 0.0, 0.0, lam, g);
    adj_entrance_misalign(lam, e);
}

/* ---- any element: forward mode on dual numbers --------------------------- */

template <int K>
__device__ __forceinline__ Lam6 adj_dual(const P6& s, const Lam6& in, const Rec& e, int nturn,
                                         const Param& pm) {
    using D = Dual<K>;
    P6T<D> r;
    r.x = D(s.x); r.px = D(s.px); r.y = D(s.y);
    r.py = D(s.py); r.dp = D(s.dp); r.ct = D(s.ct);
    r.x.d[0] = 1.0; r.px.d[1] = 1.0; r.y.d[2] = 1.0;
    r.py.d[3] = 1.0; r.dp.d[4] = 1.0; r.ct.d[5] = 1.0;
    NoRecip<D> none;
    track_element(r, none, e, nturn, pm);
    const D* rows[6] = {&r.x, &r.px, &r.y, &r.py, &r.dp, &r.ct};
    Lam6 out;
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        double a = 0.0;
#pragma unroll
        for (int i = 0; i < 6; ++i) a = fma(in.v[i], rows[i]->d[j], a);
        out.v[j] = a;
    }
    out.g = 0.0;
    if constexpr (K == 7) {
#pragma unroll
        for (int i = 0; i < 6; ++i) out.g = fma(in.v[i], rows[i]->d[6], out.g);
    }
    return out;
}

__device__ __noinline__ Lam6 adj_dual6(P6 s, Lam6 in, Rec e, int nturn) {
    return adj_dual<6>(s, in, e, nturn, Param{-1, 0.0});
}

__device__ __noinline__ Lam6 adj_dual7(P6 s, Lam6 in, Rec e, int nturn, Param pm) {
    return adj_dual<7>(s, in, e, nturn, pm);
}

__device__ __forceinline__ void adj_any(const P6& s, const P6& sx, Recip& rc, double* lam,
                                        const Rec& e, int nturn, const Param& pm, double& g) {
    switch (e.op()) {
        case ATB_OP_DRIFT: adj_pass_drift(s, rc, lam, e); return;
        case ATB_OP_IDENTITY:
            adj_exit_misalign(lam, e);
            adj_entrance_misalign(lam, e);
            return;
        case ATB_OP_APERTURE:
        case ATB_OP_QUANTDIFF: return;      /* identity for a surviving particle */
        case ATB_OP_RFCAVITY: adj_pass_rfcavity(s, lam, e, nturn); return;
        case ATB_OP_CORRECTOR:
            if (!(e.flags() & (ATB_F_THICK | ATB_F_SCALING))) {   /* px += xk, py += yk */
                adj_exit_misalign(lam, e);
                adj_entrance_misalign(lam, e);
                return;
            }
            break;
        case ATB_OP_THINMPOLE:
            if (!(e.flags() & ATB_F_SCALING)) { adj_pass_thinmpole(s, lam, e, pm, g); return; }
            break;
        case ATB_OP_STRMPOLE:
            if (adj_by_hand(e, false)) { adj_pass_multipole<false>(s, sx, rc, lam, e, pm, g); return; }
            break;
        case ATB_OP_BNDMPOLE:
            if (adj_by_hand(e, true)) { adj_pass_multipole<true>(s, sx, rc, lam, e, pm, g); return; }
            break;
        default: break;
    }
    Lam6 in;
#pragma unroll
    for (int i = 0; i < 6; ++i) in.v[i] = lam[i];
    in.g = 0.0;
    const Lam6 out = pm.k >= 0 ? adj_dual7(s, in, e, nturn, pm) : adj_dual6(s, in, e, nturn);
#pragma unroll
    for (int i = 0; i < 6; ++i) lam[i] = out.v[i];
    g += out.g;
}

/* any element, out of line: what most of a ring's elements do not need would
 * otherwise have the sweep's state spilled around every one of them */
__device__ __noinline__ Lam6 adj_rare(P6 s, P6 sx, double pn, Lam6 in, Rec e, int nturn,
                                      Param pm) {
    Recip rc;
    rc.dp = s.dp;
    rc.pn = pn;
    adj_any(s, sx, rc, in.v, e, nturn, pm, in.g);
    return in;
}

/* lambda <- J_e(s)^T lambda; g += the strength's term; sx: the exit state */
__device__ __forceinline__ void adj_element(const P6& s, const P6& sx, Recip& rc, double* lam,
                                            const Rec& e, int nturn, const Param& pm,
                                            double& g) {
    const int op = e.op(), mo = e.mo();
    const bool plain = e.opt == 0, upright = e.flags() & ATB_F_NOSKEW;
    if (op == ATB_OP_DRIFT && plain) {
        adj_drift6(s, lam, e.f(ATB_DR_LE), opd_rcp(rc, s.dp));
        return;
    }
    if (op == ATB_OP_STRMPOLE && plain && upright && adj_by_hand(e, false)) {
        if (mo == 1 && adj_multipole_mo<false, 1, false, true>(s, sx, rc, lam, e, pm, g)) return;
        if (mo == 2 && adj_multipole_mo<false, 2, false, true>(s, sx, rc, lam, e, pm, g)) return;
    }
    if (op == ATB_OP_BNDMPOLE && plain && upright && mo == 1 && adj_by_hand(e, true)) {
        if (adj_multipole_mo<true, 1, false, true>(s, sx, rc, lam, e, pm, g)) return;
    }
    Lam6 io;
#pragma unroll
    for (int i = 0; i < 6; ++i) io.v[i] = lam[i];
    io.g = g;
    io = adj_rare(s, sx, opd_rcp(rc, s.dp), io, e, nturn, pm);
#pragma unroll
    for (int i = 0; i < 6; ++i) lam[i] = io.v[i];
    g = io.g;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

/* ---- kernels ------------------------------------------------------------- */

extern "C" __global__ void __launch_bounds__(ATB_ADJ_THREADS)
atb_adjoint_forward_kernel(const AtbAdjoint A) {
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= A.np) return;
    P6 r;
    load6(A.r + 6 * p, r);
    bool lost = isnan(r.x);
    Recip rc;
    for (int tt = 0; tt < A.nturns; ++tt) {
        if (A.ckpt && tt % A.stride == 0)
            store6(A.ckpt + 6 * ((long long)(tt / A.stride) * A.ld + p), r);
        if (lost || (A.skip_last && tt == A.nturns - 1)) continue;
        const int nturn = A.turn0 + tt;
        for (int ei = 0; ei < A.nelem; ++ei) {
            if (A.scratch)
                store6(A.scratch + 6 * (((long long)tt * A.nelem + ei) * A.ld + p), r);
            track_element(r, rc, adj_rec(A, ei), nturn, adj_param(A, ei));
            if (is_bad(r)) {                  /* pyat/at.c:115-139 */
                lost = true;
                break;
            }
        }
        if (lost) {
            r.x = nan_d(); r.px = 0.0; r.y = 0.0; r.py = 0.0; r.dp = 0.0; r.ct = 0.0;
        }
    }
    store6(A.r + 6 * p, r);
    if (A.lost) A.lost[p] = lost ? 1 : 0;
}

extern "C" __global__ void __launch_bounds__(ATB_ADJ_THREADS, ATB_ADJ_MIN_BLOCKS)
atb_adjoint_turn_kernel(const AtbAdjoint A) {
    /* the block's strength gradient (nparam words) */
    extern __shared__ double sg[];
    for (int q = threadIdx.x; q < A.nparam; q += blockDim.x) sg[q] = 0.0;
    __syncthreads();
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = p < A.np;
    const long long np = A.np;
    P6 exit;                      /* leaving the element at hand */
    double lam[6];
    bool live = false;
    if (in) {
        /* a particle lost during the turn enters the next one as NaN */
        live = !isnan(__ldg(A.ckpt + 6 * p));
        load6(A.next + 6 * p, exit);
        live &= !isnan(exit.x);
#pragma unroll
        for (int i = 0; i < 6; ++i) lam[i] = A.lam[6 * p + i];
#pragma unroll
        for (int i = 0; i < 6; ++i) live &= isfinite(lam[i]);
    }
    /* an element's entry state is asked for while the one behind it is worked
       on: it comes from HBM */
    P6 ahead;
    Recip rc;
    if (live && A.nelem > 0) load6(A.scratch + 6 * ((long long)(A.nelem - 1) * np + p), ahead);
    for (int ei = A.nelem - 1; ei >= 0; --ei) {
        const Param pm = adj_param(A, ei);
        double g = 0.0;
        if (live) {
            const P6 se = ahead;
            if (ei > 0) load6(A.scratch + 6 * ((long long)(ei - 1) * np + p), ahead);
            adj_element(se, exit, rc, lam, adj_rec(A, ei), A.turn0, pm, g);
            exit = se;
        }
        if (pm.k >= 0) {                      /* the same for the whole block */
            g = warp_sum(g);
            if ((threadIdx.x & 31) == 0) atomicAdd(&sg[A.pelem[ei]], g);
        }
    }
    if (in) {
        const double nan = nan_d();
#pragma unroll
        for (int i = 0; i < 6; ++i) A.lam[6 * p + i] = live ? lam[i] : nan;
    }
    __syncthreads();
    for (int q = threadIdx.x; q < A.nparam; q += blockDim.x)
        if (sg[q] != 0.0) atomicAdd(&A.gparam[q], sg[q]);
}

}  // namespace atb

#endif  // ATB_ADJOINT_KERNEL_CUH
