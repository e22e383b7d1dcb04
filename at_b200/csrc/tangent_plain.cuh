/*
 * The tangent kernel of lattices whose elements all have a hand-written
 * derivative (atb_tangent_by_hand of atb_table.h): drifts, non-radiating
 * magnets, thin multipoles and correctors, cavities, apertures.
 *
 * The general tangent kernel runs every operation on dual numbers of seven
 * slots.  Here a magnet's steps carry the particle (by the exact kernels' own
 * operations) and the columns of the magnet's Jacobian with respect to its
 * entrance (x, px, y, py, delta): a drift and kick cost two or three fused
 * operations a column where the dual numbers spend about thirty a slot, delta
 * and ct need no column of their own (delta is constant, ct feeds nothing),
 * and in upright magnets up to the quadrupole the planes do not mix.  The
 * tangent map J(s) = d r(s) / d r0 of the particle waits in shared memory and
 * is updated by the magnet's matrix once per magnet.
 *
 * Bound: the FP64 pipe when the SMs are full, dependent latency below that
 * (one warp a scheduler up to 19,000 particles).  One turn of the FODO ring with
 * 128 strengths: 16,411 particles 1.58 ms (4.6 on dual numbers), 65,536
 * particles 3.83 ms (12.9).  168 registers and three blocks an SM: with 128
 * and four the columns spill (3 KB of stores), with 255 and two the larger set
 * takes 3 % longer.
 */
#ifndef ATB_TANGENT_PLAIN_CUH
#define ATB_TANGENT_PLAIN_CUH

#include "track_kernel.cuh"
#include "atb_solve6.cuh"

namespace atb {

/* The particle's tangent map in shared memory, entry (i, j) at
 * base[(6 i + j) * ATB_TANGENT_THREADS]: a warp's accesses are consecutive. */
struct TanMap {
    double* base;
    __device__ __forceinline__ double& at(int i, int j) const {
        return base[(6 * i + j) * ATB_TANGENT_THREADS];
    }
};

/* One column of a magnet's Jacobian (its delta entry is that of the entrance
 * variable). */
struct TanCol {
    double x, px, y, py, ct;
};

/* The columns: with respect to x, px, y, py, delta (c[0..4]) and to the
 * differentiated strength (c[5]).  In a decoupled magnet (DEC) the x columns
 * have no y entries and the y columns no x entries.  They hold what the magnet
 * adds to a drift as long as the stages so far: to 1 in dx/dx, dpx/dpx, dy/dy,
 * dpy/dpy, to the length s (over 1 + delta) in dx/dpx and dy/dpy, to sx and sy
 * in dct/dpx and dct/dpy.  Equal magnets round alike, so that the errors of
 * their Jacobians add up over a ring; with whole entries, rounded at the size
 * of one in every stage, the dispersion and ct terms of the FODO ring were off
 * by 1.4 times what the dual numbers leave. */
struct TanCols {
    TanCol c[6];
    double s, sx, sy;
};
__device__ __forceinline__ double tan_x(const TanCols& t, int j) {
    return j == 0 ? 1.0 + t.c[0].x : j == 1 ? t.s + t.c[1].x : t.c[j].x;
}
__device__ __forceinline__ double tan_y(const TanCols& t, int j) {
    return j == 2 ? 1.0 + t.c[2].y : j == 3 ? t.s + t.c[3].y : t.c[j].y;
}

template <bool DEC>
__device__ __forceinline__ constexpr bool tan_has_x(int j) { return !DEC || j < 2 || j > 3; }
template <bool DEC>
__device__ __forceinline__ constexpr bool tan_has_y(int j) { return !DEC || j > 1; }

/* d/dz of the field F(z) = sum (B_n + i A_n) z^n, with the coefficients of a
 * Poly holder */
template <int MO, bool SKEW>
__device__ __forceinline__ void tan_prime(const Poly<MO, SKEW>& p, double x, double y, double& dr,
                                          double& di) {
    if constexpr (MO <= 0) {
        dr = 0.0;
        di = 0.0;
    } else {
        dr = (double)MO * p.b[MO];
        di = SKEW ? (double)MO * p.a[SKEW ? MO : 0] : 0.0;
#pragma unroll
        for (int n = MO - 1; n >= 1; --n) {
            const double an = SKEW ? (double)n * p.a[SKEW ? n : 0] : 0.0;
            const double t = fma(dr, x, fma(-di, y, (double)n * p.b[n]));
            di = fma(di, x, fma(dr, y, an));
            dr = t;
        }
    }
}
__device__ __forceinline__ void tan_prime(const Poly<-1>& p, double x, double y, double& dr,
                                          double& di) {
    dr = 0.0;
    di = 0.0;
    if (p.mo <= 0) return;
    dr = (double)p.mo * (p.sk == p.mo ? p.kv : p.b[p.mo]);
    di = (double)p.mo * p.a[p.mo];
    for (int n = p.mo - 1; n >= 1; --n) {
        const double t = fma(dr, x, fma(-di, y, (double)n * (p.sk == n ? p.kv : p.b[n])));
        di = fma(di, x, fma(dr, y, (double)n * p.a[n]));
        dr = t;
    }
}

/* z^k = (x + i y)^k */
__device__ __forceinline__ void tan_zpow(double x, double y, int k, double& zr, double& zi) {
    zr = x;
    zi = y;
    for (int i = 1; i < k; ++i) {
        const double t = fma(zr, x, -zi * y);
        zi = fma(zr, y, zi * x);
        zr = t;
    }
}

/* The columns through `f` (1 or 2) equal drifts of normalised length nl whose
 * increments at (px, py) are d: pe and pb are 1/(1+delta) of the element's
 * entry (in nl; 0 keeps that dependence out of the delta column) and of its
 * body. */
template <bool DEC, bool HASK>
__device__ __forceinline__ void tan_drift(const P6& r, TanCols& t, const DriftInc& d, double f,
                                          double nl, double pe, double pb) {
    const double n = f * nl, w = n * pb;
    const double tx = w * r.px, ty = w * r.py;
#pragma unroll
    for (int j = 0; j < (HASK ? 6 : 5); ++j) {
        TanCol& c = t.c[j];
        if (tan_has_x<DEC>(j)) {
            c.x = fma(n, c.px, c.x);
            c.ct = fma(tx, c.px, c.ct);
        }
        if (tan_has_y<DEC>(j)) {
            c.y = fma(n, c.py, c.y);
            c.ct = fma(ty, c.py, c.ct);
        }
    }
    t.s += n;
    t.sx += tx;
    t.sy += ty;
    TanCol& e = t.c[4];
    const double fe = f * pe;
    e.x = fma(-fe, d.x, e.x);
    e.y = fma(-fe, d.y, e.y);
    e.ct = fma(-fma(f, pb, fe), d.ct, e.ct);
}

/* The columns through the kick of length L at (x, y) (strthinkick,
 * bndthinkick). */
template <bool DEC, bool BEND, bool HASK, class PL>
__device__ __forceinline__ void tan_kick(const P6& r, TanCols& t, const PL& pl, int pk, double L,
                                         double irho, double lirho) {
    double dr, di;
    tan_prime(pl, r.x, r.y, dr, di);
    const double ay = L * dr, b = L * di;
    const double li = BEND ? L * irho : 0.0;
    const double ax = BEND ? fma(li, irho, ay) : ay;
#pragma unroll
    for (int j = 0; j < (HASK ? 6 : 5); ++j) {
        TanCol& c = t.c[j];
        const double x = tan_x(t, j), y = tan_y(t, j);
        if (tan_has_x<DEC>(j)) {
            c.px = fma(-ax, x, c.px);
            if (BEND) c.ct = fma(lirho, x, c.ct);
        }
        if (tan_has_y<DEC>(j)) c.py = fma(ay, y, c.py);
        if (!DEC) {
            c.px = fma(b, y, c.px);
            c.py = fma(b, x, c.py);
        }
    }
    if (BEND) t.c[4].px += li;
    if (HASK) {
        double zr, zi;
        tan_zpow(r.x, r.y, pk, zr, zi);
        t.c[5].px = fma(-L, zr, t.c[5].px);
        t.c[5].py = fma(L, zi, t.c[5].py);
    }
}

/* The integration steps of a non-radiating magnet: the particle by the
 * operations of multipole_steps_rn (the plain expressions again if an operand
 * is out of range: its columns do not depend on those last bits), the columns
 * beside it. */
template <bool BEND, int MO, bool SKEW, bool HASK>
__device__ __forceinline__ void tan_steps(P6& r, TanCols& t, const Rec& e, const Param& pm,
                                          double pb, double pe, double nl1, double nl2,
                                          double irho, int ns) {
    if (ns <= 0) return;
    constexpr bool DEC = MO == 0 || (MO == 1 && !SKEW);
    const double K1 = e.f(ATB_SM_K1), K2 = e.f(ATB_SM_K2);
    const double k1i = BEND ? e.f(ATB_BM_K1IRHO) : 0.0, k2i = BEND ? e.f(ATB_BM_K2IRHO) : 0.0;
    const int mo = e.mo();
    const double* A = e.p + (BEND ? ATB_BM_POLY : ATB_SM_POLY);
    Poly<MO, SKEW> pl;
    pl.load(A, A + mo + 1, mo);
    if (HASK) pl.set_param(pm.k, pm.v);
    const P6 in = r;
    const double o = 1.0 + r.dp;
    const double od2 = 2.0 * o, hp = 0.5 * pb;
    bool ok = (e.flags() & ATB_F_RN) && rn_coords_fit(r.x, r.px, r.y, r.py) && rn_opd_constant(o);
    DriftInc d = fastdrift_inc(r, nl1, od2, hp);
    tan_drift<DEC, HASK>(r, t, d, 1.0, nl1, pe, pb);
    add_drift(r, d);
    for (int m = 1;; ++m) {
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
            const double K = h ? K2 : K1, ki = h ? k2i : k1i;
            tan_kick<DEC, BEND, HASK>(r, t, pl, pm.k, K, irho, ki);
            if (BEND) bndthinkick(r, pl, K, irho, ki); else strthinkick(r, pl, K);
            d = fastdrift_inc(r, nl2, od2, hp);
            tan_drift<DEC, HASK>(r, t, d, 1.0, nl2, pe, pb);
            add_drift(r, d);
        }
        tan_kick<DEC, BEND, HASK>(r, t, pl, pm.k, K1, irho, k1i);
        if (BEND) bndthinkick(r, pl, K1, irho, k1i); else strthinkick(r, pl, K1);
        d = fastdrift_inc(r, nl1, od2, hp);
        tan_drift<DEC, HASK>(r, t, d, m == ns ? 1.0 : 2.0, nl1, pe, pb);
        add_drift(r, d);
        if (m == ns) break;
        add_drift(r, d);
    }
    ok &= rn_ordinary(r.ct);
    if (!ok) r = multipole_steps_call<BEND, false>(in, e, pm, nl1, nl2);
}

/* fy of edge_fringe (methods other than 3) and its derivative with respect to
 * delta */
__device__ __forceinline__ void tan_edge(const P6& r, const Rec& e, double irho, int w_edge,
                                         int method, bool fc0, double& fy, double& dfy) {
    const double edge = e.f(w_edge), fc = e.f(w_edge + 1), fy_c = e.f(w_edge + 3);
    const double opd = 1.0 + r.dp;
    fy = fy_c;
    dfy = 0.0;
    if (!fc0) {
        const double a = edge - fc / opd;
        const double tn = tan(a);
        if (a != edge) fy = irho * tn;
        dfy = irho * fma(tn, tn, 1.0) * fc / (opd * opd);
    }
    if (method == ATB_BM_2) {
        fy = fy / opd;
        dfy = (dfy - fy) / opd;
    }
}

/* The column of a magnet's Jacobian with respect to the momentum of its entry,
 * through the drift lengths L/(1+delta) alone, from the entrance edge to the
 * exit edge.  A dense entrance rotation mixes delta, so that it is not the
 * body's delta; otherwise the delta column holds it.  Out of line, its results
 * in the frame, so that the rare case takes no registers. */
struct TanMix {
    double entry[6];          /* d delta_entry / d r0 */
    TanCol n;
};
__device__ __noinline__ void tan_mix_entry(TanMap J, TanMix* mix) {
    for (int j = 0; j < 6; ++j) mix->entry[j] = J.at(4, j);
}
__device__ __noinline__ void tan_mix_exit(TanMap J, const TanMix* mix) {
    const TanCol n = mix->n;
    for (int j = 0; j < 6; ++j) {
        const double d = mix->entry[j];
        J.at(0, j) = fma(n.x, d, J.at(0, j));
        J.at(1, j) = fma(n.px, d, J.at(1, j));
        J.at(2, j) = fma(n.y, d, J.at(2, j));
        J.at(3, j) = fma(n.py, d, J.at(3, j));
        J.at(5, j) = fma(n.ct, d, J.at(5, j));
    }
}
__device__ __noinline__ void tan_mix_body(P6 r, Rec e, Param pm, double pe, double nl1,
                                          double nl2, bool bend, TanMix* mix) {
    const int mo = e.mo();
    const double* A = e.p + (bend ? ATB_BM_POLY : ATB_SM_POLY);
    Poly<-1> pl;
    pl.load(A, A + mo + 1, mo);
    if (pm.k >= 0) pl.set_param(pm.k, pm.v);
    const double irho = bend ? e.f(ATB_BM_IRHO) : 0.0;
    const double pb = 1.0 / (1.0 + r.dp);
    TanCols t;
    TanCol& c = t.c[4];
    c = TanCol{0.0, 0.0, 0.0, 0.0, 0.0};
    for (int m = 0; m < e.nsteps(); ++m) {
        for (int i = 0; i < 4; ++i) {
            const double nl = i == 0 || i == 3 ? nl1 : nl2, w = nl * pb;
            const double s = fma(r.px, r.px, r.py * r.py);
            c.x = fma(nl, fma(-pe, r.px, c.px), c.x);
            c.y = fma(nl, fma(-pe, r.py, c.py), c.y);
            c.ct = fma(w, fma(r.px, c.px, fma(r.py, c.py, -0.5 * pe * s)), c.ct);
            r.x = fma(nl, r.px, r.x);
            r.y = fma(nl, r.py, r.y);
            if (i == 3) break;
            const double K = i == 1 ? e.f(ATB_SM_K2) : e.f(ATB_SM_K1);
            double dr, di;
            tan_prime(pl, r.x, r.y, dr, di);
            c.px = fma(-K, fma(dr + irho * irho, c.x, -di * c.y), c.px);
            c.py = fma(K, fma(di, c.x, dr * c.y), c.py);
            c.ct = fma(K * irho, c.x, c.ct);
            if (bend) bndthinkick(r, pl, K, irho, K * irho); else strthinkick(r, pl, K);
        }
    }
    if (bend) {
        double fy, dfy;
        tan_edge(r, e, irho, ATB_BM_EOUT, (int)((e.flags() >> ATB_F_BM_OUT_SHIFT) & ATB_F_BM_MASK),
                 e.flags() & ATB_F_FC0_OUT, fy, dfy);
        c.px = fma(e.f(ATB_BM_FXOUT), c.x, c.px);
        c.py = fma(-fy, c.y, c.py);
    }
    mix->n = c;
}

/* J <- R J of a misalignment rotation (mult_r) */
__device__ __forceinline__ void tan_rotate(const TanMap& J, const double* m, bool dense) {
#pragma unroll 1
    for (int j = 0; j < 6; ++j) {
        double v[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) v[i] = J.at(i, j);
        if (dense) {
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                double s = 0.0;
#pragma unroll
                for (int k = 0; k < 6; ++k) s = fma(m[i + 6 * k], v[k], s);
                J.at(i, j) = s;
            }
        } else {
            J.at(0, j) = fma(m[0], v[0], m[1] * v[2]);
            J.at(1, j) = fma(m[2], v[1], m[3] * v[3]);
            J.at(2, j) = fma(m[4], v[0], m[5] * v[2]);
            J.at(3, j) = fma(m[6], v[1], m[7] * v[3]);
        }
    }
}
__device__ __forceinline__ void tan_rotate(double* g, const double* m, bool dense) {
    double v[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) v[i] = g[i];
    if (dense) {
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            g[i] = 0.0;
#pragma unroll
            for (int k = 0; k < 6; ++k) g[i] = fma(m[i + 6 * k], v[k], g[i]);
        }
    } else {
        g[0] = fma(m[0], v[0], m[1] * v[2]);
        g[1] = fma(m[2], v[1], m[3] * v[3]);
        g[2] = fma(m[4], v[0], m[5] * v[2]);
        g[3] = fma(m[6], v[1], m[7] * v[3]);
    }
}

__device__ __forceinline__ void tan_entrance(P6& r, const TanMap& J, const Rec& e) {
    if (!e.opt) return;
    entrance_misalign(r, e);
    if (const double* r1 = e.blk(ATB_OPT_R1)) tan_rotate(J, r1, e.flags() & ATB_F_R1_DENSE);
    apertures(r, e);
}

/* g: the strength's column, or null */
__device__ __forceinline__ void tan_exit(P6& r, const TanMap& J, const Rec& e, double* g) {
    if (!e.opt) return;
    apertures(r, e);
    exit_misalign(r, e);
    if (const double* r2 = e.blk(ATB_OPT_R2)) {
        tan_rotate(J, r2, e.flags() & ATB_F_R2_DENSE);
        if (g) tan_rotate(g, r2, e.flags() & ATB_F_R2_DENSE);
    }
}

/* J through a drift of length L at the particle's (px, py) */
__device__ __forceinline__ void tan_drift6(P6& r, const TanMap& J, double L, double pn) {
    const double nl = L * pn, w = nl * pn;
    const double tx = w * r.px, ty = w * r.py;
    const double tc = -w * pn * fma(r.px, r.px, r.py * r.py);
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        const double dpx = J.at(1, j), dpy = J.at(3, j), dd = J.at(4, j);
        J.at(0, j) += fma(nl, dpx, -(tx * dd));
        J.at(2, j) += fma(nl, dpy, -(ty * dd));
        J.at(5, j) += fma(tx, dpx, fma(ty, dpy, tc * dd));
    }
    drift6_pn<false>(r, L, pn);
}

__device__ __forceinline__ void tan_rf(P6& r, const TanMap& J, const Rec& e, int nturn) {
    if (!(e.flags() & ATB_F_NV)) return;
    const double nv = e.f(ATB_RF_NV), tf = e.f(ATB_RF_TF), lag = e.f(ATB_RF_LAG);
    const double a = tf * ((r.ct - lag) / ATB_C0 - e.f(ATB_RF_HT) * (double)nturn) -
                     e.f(ATB_RF_PHI);
    const double k = -nv * cos(a) * (tf / ATB_C0);
#pragma unroll
    for (int j = 0; j < 6; ++j) J.at(4, j) = fma(k, J.at(5, j), J.at(4, j));
    rf_kick(r, e, nturn);
}

/* A non-radiating magnet; HASK: g receives d r_out / d K of the magnet alone. */
template <bool BEND, bool HASK>
__device__ __forceinline__ void tan_magnet(P6& r, Recip& rc, const TanMap& J, const Rec& e,
                                           const Param& pm, double* g) {
    const uint32_t fl = e.flags();
    const double dp0 = r.dp, pe = opd_rcp(rc, r.dp);
    const double nl1 = e.f(ATB_SM_L1) * pe, nl2 = e.f(ATB_SM_L2) * pe;
    const bool mixed = (fl & ATB_F_R1_DENSE) && e.blk(ATB_OPT_R1);
    TanMix mix;
    if (mixed) tan_mix_entry(J, &mix);
    tan_entrance(r, J, e);
    const double pb = r.dp == dp0 ? pe : 1.0 / (1.0 + r.dp);
    const double pc = mixed ? 0.0 : pe;
    TanCols t;
#pragma unroll
    for (int j = 0; j < 6; ++j) t.c[j] = TanCol{0.0, 0.0, 0.0, 0.0, 0.0};
    t.s = t.sx = t.sy = 0.0;
    double irho = 0.0;
    if (BEND) {
        irho = e.f(ATB_BM_IRHO);
        double fy, dfy;
        const int m_in = (int)((fl >> ATB_F_BM_IN_SHIFT) & ATB_F_BM_MASK);
        tan_edge(r, e, irho, ATB_BM_EIN, m_in, fl & ATB_F_FC0_IN, fy, dfy);
        t.c[0].px = e.f(ATB_BM_FXIN);
        t.c[2].py = -fy;
        t.c[4].py = -r.y * dfy;
        edge_fringe<false>(r, irho, e.f(ATB_BM_EIN), e.f(ATB_BM_FCIN), e.f(ATB_BM_FXIN),
                           e.f(ATB_BM_FYIN), m_in, fl & ATB_F_FC0_IN, 1.0);
    }
    if (mixed) tan_mix_body(r, e, pm, pe, nl1, nl2, BEND, &mix);
    const int ns = e.nsteps();
#define ATB_TAN_STEPS(MO, SKEW) \
    tan_steps<BEND, MO, SKEW, HASK>(r, t, e, pm, pb, pc, nl1, nl2, irho, ns)
    const bool upright = fl & ATB_F_NOSKEW;
    const int mo = e.mo();
    if (mo == 0 && !HASK) ATB_TAN_STEPS(0, true);
    else if (mo == 1 && upright) ATB_TAN_STEPS(1, false);
    else if (mo == 2 && upright) ATB_TAN_STEPS(2, false);
    else if (mo == 3 && upright) ATB_TAN_STEPS(3, false);
    else ATB_TAN_STEPS(-1, true);
#undef ATB_TAN_STEPS
    if (BEND) {
        double fy, dfy;
        const int m_out = (int)((fl >> ATB_F_BM_OUT_SHIFT) & ATB_F_BM_MASK);
        tan_edge(r, e, irho, ATB_BM_EOUT, m_out, fl & ATB_F_FC0_OUT, fy, dfy);
        const double fx = e.f(ATB_BM_FXOUT);
#pragma unroll
        for (int j = 0; j < (HASK ? 6 : 5); ++j) {
            t.c[j].px = fma(fx, tan_x(t, j), t.c[j].px);
            t.c[j].py = fma(-fy, tan_y(t, j), t.c[j].py);
        }
        t.c[4].py = fma(-r.y, dfy, t.c[4].py);
        edge_fringe<false>(r, irho, e.f(ATB_BM_EOUT), e.f(ATB_BM_FCOUT), e.f(ATB_BM_FXOUT),
                           e.f(ATB_BM_FYOUT), m_out, fl & ATB_F_FC0_OUT, -1.0);
    }
    if (HASK) {
        g[0] = t.c[5].x; g[1] = t.c[5].px; g[2] = t.c[5].y;
        g[3] = t.c[5].py; g[4] = 0.0; g[5] = t.c[5].ct;
    }
    /* J <- M J */
#pragma unroll 2
    for (int j = 0; j < 6; ++j) {
        double v[5], s[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) v[k] = J.at(k, j);
        s[0] = t.s * v[1];
        s[1] = 0.0;
        s[2] = t.s * v[3];
        s[3] = 0.0;
        s[4] = fma(t.sx, v[1], t.sy * v[3]);
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            s[0] = fma(t.c[k].x, v[k], s[0]);
            s[1] = fma(t.c[k].px, v[k], s[1]);
            s[2] = fma(t.c[k].y, v[k], s[2]);
            s[3] = fma(t.c[k].py, v[k], s[3]);
            s[4] = fma(t.c[k].ct, v[k], s[4]);
        }
        J.at(0, j) = v[0] + s[0]; J.at(1, j) = v[1] + s[1]; J.at(2, j) = v[2] + s[2];
        J.at(3, j) = v[3] + s[3]; J.at(5, j) += s[4];
    }
    if (mixed) tan_mix_exit(J, &mix);
    tan_exit(r, J, e, HASK ? g : nullptr);
}

/* ThinMPolePass without field scaling */
__device__ __forceinline__ void tan_thinmpole(P6& r, const TanMap& J, const Rec& e,
                                              const Param& pm, double* g) {
    const int mo = e.mo();
    const double* A = e.p + ATB_TM_POLY;
    Poly<-1> pl;
    pl.load(A, A + mo + 1, mo);
    if (pm.k >= 0) pl.set_param(pm.k, pm.v);
    const double bax = e.f(ATB_TM_BAX), bay = e.f(ATB_TM_BAY);
    tan_entrance(r, J, e);
    double dr, di;
    tan_prime(pl, r.x, r.y, dr, di);
#pragma unroll 1
    for (int j = 0; j < 6; ++j) {
        const double dx = J.at(0, j), dy = J.at(2, j), dd = J.at(4, j);
        J.at(1, j) += fma(-dr, dx, fma(di, dy, bax * dd));
        J.at(3, j) += fma(di, dx, fma(dr, dy, -bay * dd));
        J.at(5, j) += fma(-bax, dx, bay * dy);
    }
    if (pm.k >= 0) {
        double zr, zi;
        tan_zpow(r.x, r.y, pm.k, zr, zi);
        g[0] = g[2] = g[4] = g[5] = 0.0;
        g[1] = -zr;
        g[3] = zi;
    }
    strthinkick(r, pl, 1.0);
    r.px += bax * r.dp;
    r.py -= bay * r.dp;
    r.ct -= bax * r.x - bay * r.y;
    /* the reference checks this element's apertures at the entrance only */
    exit_misalign(r, e);
    if (const double* r2 = e.blk(ATB_OPT_R2)) {
        tan_rotate(J, r2, e.flags() & ATB_F_R2_DENSE);
        if (pm.k >= 0) tan_rotate(g, r2, e.flags() & ATB_F_R2_DENSE);
    }
}

/* One element on the particle and its tangent map. */
__device__ __forceinline__ void tan_element(P6& r, Recip& rc, const TanMap& J, const Rec& e,
                                            int nturn, const Param& pm, double* g) {
    switch (e.op()) {
        case ATB_OP_DRIFT:
            tan_entrance(r, J, e);
            tan_drift6(r, J, e.f(ATB_DR_LE), opd_rcp(rc, r.dp));
            tan_exit(r, J, e, nullptr);
            break;
        case ATB_OP_STRMPOLE:
            if (pm.k >= 0) tan_magnet<false, true>(r, rc, J, e, pm, g);
            else tan_magnet<false, false>(r, rc, J, e, pm, g);
            break;
        case ATB_OP_BNDMPOLE:
            if (pm.k >= 0) tan_magnet<true, true>(r, rc, J, e, pm, g);
            else tan_magnet<true, false>(r, rc, J, e, pm, g);
            break;
        case ATB_OP_IDENTITY:
            tan_entrance(r, J, e);
            tan_exit(r, J, e, nullptr);
            break;
        case ATB_OP_CORRECTOR:             /* thin, without field scaling */
            tan_entrance(r, J, e);
            r.px += e.f(ATB_CO_XK);
            r.py += e.f(ATB_CO_YK);
            exit_misalign(r, e);
            if (const double* r2 = e.blk(ATB_OPT_R2))
                tan_rotate(J, r2, e.flags() & ATB_F_R2_DENSE);
            break;
        case ATB_OP_THINMPOLE: tan_thinmpole(r, J, e, pm, g); break;
        case ATB_OP_RFCAVITY:
            if (e.flags() & ATB_F_THICK) tan_drift6(r, J, e.f(ATB_RF_HALF), opd_rcp(rc, r.dp));
            tan_rf(r, J, e, nturn);
            if (e.flags() & ATB_F_THICK) tan_drift6(r, J, e.f(ATB_RF_HALF), opd_rcp(rc, r.dp));
            break;
        case ATB_OP_APERTURE: check_rect(r, e.p + ATB_AP_LIM); break;
        default: break;                    /* quantum diffusion: the identity */
    }
}

extern "C" __global__ void __launch_bounds__(ATB_TANGENT_THREADS, 3)
atb_tangent_plain_kernel(const AtbTangent A) {
    __shared__ double maps[36 * ATB_TANGENT_THREADS];
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= A.np) return;
    const long long np = A.np;
    const TanMap J{maps + threadIdx.x};
#pragma unroll 1
    for (int i = 0; i < 6; ++i) {
#pragma unroll
        for (int j = 0; j < 6; ++j) J.at(i, j) = i == j ? 1.0 : 0.0;
    }
    P6 r;
    load6(A.r + 6 * p, r);
    Recip rc;
    bool lost = false;
    for (int tt = 0; tt < A.nturns && !lost; ++tt) {
        for (int ei = 0; ei < A.nelem; ++ei) {
            Rec e;
            e.p = A.table + A.elem_off[ei];
            const uint64_t* hp = reinterpret_cast<const uint64_t*>(e.p);
            e.hdr = hp[0];
            e.opt = hp[1];
            const int q = A.pelem ? A.pelem[ei] : -1;
            Param pm{-1, 0.0};
            if (q >= 0) { pm.k = A.porder[q]; pm.v = A.pvalue[q]; }
            double g[6];
            if (!isnan(r.x)) tan_element(r, rc, J, e, A.turn0 + tt, pm, g);
            if (is_bad(r)) {          /* pyat/at.c:115-139 */
                lost = true;
                break;
            }
            if (q >= 0) {
                double M[6][7], w[6];
#pragma unroll
                for (int i = 0; i < 6; ++i) {
#pragma unroll
                    for (int j = 0; j < 6; ++j) M[i][j] = J.at(i, j);
                    M[i][6] = g[i];
                }
                solve6(M, w);
                double* u = A.grad + 6LL * q * np + p;
#pragma unroll
                for (int i = 0; i < 6; ++i) u[i * np] = tt ? u[i * np] + w[i] : w[i];
            }
        }
    }

    const double nan = nan_d();
    for (int q = 0; q < A.nparam; ++q) {
        double* gq = A.grad + 6LL * q * np + p;
        double u[6];
#pragma unroll
        for (int j = 0; j < 6; ++j) u[j] = lost || A.nturns <= 0 ? 0.0 : gq[j * np];
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            double s = 0.0;
#pragma unroll
            for (int j = 0; j < 6; ++j) s += J.at(i, j) * u[j];
            gq[i * np] = lost ? nan : s;
        }
    }
#pragma unroll 1
    for (int i = 0; i < 6; ++i) {
#pragma unroll
        for (int j = 0; j < 6; ++j) A.jac[36 * p + 6 * i + j] = lost ? nan : J.at(i, j);
    }
    if (lost) { r.x = nan; r.px = 0.0; r.y = 0.0; r.py = 0.0; r.dp = 0.0; r.ct = 0.0; }
    store6(A.r + 6 * p, r);
    if (A.lost) A.lost[p] = lost ? 1 : 0;
}

}  // namespace atb

#endif  // ATB_TANGENT_PLAIN_CUH
