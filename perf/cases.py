"""The workloads whose time is watched: tracking calls, batches and derivatives.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare(case, seed)`` makes what a user's program holds before the call,
``run(state)`` is one pass through the public entry points, ``work(case)``
what a pass cannot do without, and ``exact(case, seed)`` the same results from
plain numpy or torch in 64 bits.

The lattices are the package's own seeded rings: the 32-cell FODO ring (385
elements, with and without radiation) and the large ring (1954 elements,
misaligned, with and without radiation).
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from at_b200 import diff, flops, gpupass, rings
from at_b200.batch import BatchTracker
from at_b200.engine import Engine
from at_b200.lattice import compile_lattice


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _track(name, ring, n, turns, beam="bunch", mode="exact", losses=False, refs=0, reuse=True):
    """A call of ``gpupass`` on host arrays: ``n`` particles of a Gaussian
    bunch or an aperture grid, ``refs`` snapshot points per turn, ``reuse``
    as in the call."""
    return dict(name=name, kind="track", ring=ring, n=n, turns=turns, beam=beam, mode=mode,
                losses=losses, refs=refs, reuse=reuse)


def listed():
    return [
        # a step of a closed-orbit search: a handful of particles, one turn,
        # the lattice kept from call to call
        _track("orbit_step", "large", 7, 1),
        # the drop-in as pyat's lattice_track calls it by default: the lattice
        # is read again on every call
        _track("plain_call", "large", 200, 1, reuse=False),
        # turn-by-turn signals of a few particles (tunes, phase portraits)
        _track("turn_by_turn", "fodo", 21, 64, refs=1),
        # the FODO workload: 10,000 particles over many turns, losses recorded
        _track("fodo_bunch", "fodo", 10000, 100, losses=True),
        # many particles on the small ring, the fast arithmetic, a ragged size
        _track("fodo_fast", "fodo", 100003, 10, mode="fast", losses=True),
        # a dynamic-aperture scan: a grid of particles, most of them lost
        _track("aperture_scan", "large", 861, 12, beam="grid", losses=True),
        # beam-position monitors: snapshots at 32 places of every turn
        _track("monitors", "fodo", 10007, 10, refs=32),
        # the large ring's bunch resident on the GPU, exact arithmetic: where
        # most of a tracking study's GPU time goes
        dict(name="large_resident", kind="resident", ring="large", n=1000000, turns=2,
             mode="exact"),
        # the same ring from host arrays, the fast arithmetic, a ragged size
        _track("large_fast", "large", 200003, 1, mode="fast", losses=True),
        # error-seeded variants of the large ring (aperture grids), one launch
        dict(name="variants", kind="batch", jobs=8, n=4096, turns=10),
        # reverse mode: the gradient of a scalar of the final coordinates with
        # respect to the initial ones and to 128 strengths, forward + backward
        dict(name="adjoint", kind="adjoint", n=65536, turns=3),
        # forward mode: every particle's Jacobian and strength derivatives
        dict(name="tangent", kind="tangent", n=16411, turns=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["track"] * 6 + ["resident", "batch", "adjoint", "tangent"])
    if kind == "tangent":
        return dict(kind=kind, n=_log(rng, 1, 40000), turns=rng.randint(1, 3))
    if kind == "adjoint":
        return dict(kind=kind, n=_log(rng, 1, 100000), turns=rng.randint(1, 4))
    if kind == "batch":
        return dict(kind=kind, jobs=rng.randint(2, 10), n=_log(rng, 256, 8192),
                    turns=rng.randint(2, 12))
    ring = rng.choice(["fodo", "fodo_rad", "large", "large", "large_plain"])
    most = 400000 if ring.startswith("large") else 2000000
    mode = rng.choice(["exact", "exact", "fast"])
    if kind == "resident":
        n = _log(rng, 1000, most)
        return dict(kind=kind, ring=ring, n=n, turns=_turns(rng, ring, n), mode=mode)
    n = _log(rng, 1, 300000)
    beam = "grid" if ring.startswith("large") and mode == "exact" and rng.random() < 0.25 \
        else "bunch"
    turns = _turns(rng, ring, n)
    refs = rng.choice([0, 0, 1, 32])
    if n * turns * refs > 4000000:
        refs = 0
    c = _track("", ring, n, turns, beam, mode, rng.random() < 0.5, refs, rng.random() < 0.85)
    del c["name"]
    return c


def _turns(rng, ring, n):
    """Turns such that a pass stays below the largest listed one."""
    long, per_turn = (12, 2000000) if ring.startswith("large") else (64, 16000000)
    return max(1, min(_log(rng, 1, long), per_turn // n))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _ring(name):
    if name == "fodo":
        return rings.fodo_ring()
    if name == "fodo_rad":
        return rings.radiating(rings.fodo_ring())
    if name.startswith("variant"):
        return rings.large_ring_variant(int(name[7:]))
    return rings.large_ring(radiation=name != "large_plain")


@functools.lru_cache(maxsize=None)
def _table(name):
    ring = _ring(name)
    cl = compile_lattice(ring, ring.energy, ring.particle.rest_energy)
    return cl, float(flops.flops_per_particle_turn(cl)[0])


def _particles(ring, beam, n, seed):
    if beam == "grid":
        return rings.da_grid(n, seed)
    if ring.startswith("fodo"):
        return rings.gaussian(n, seed=seed)
    return rings.large_ring_bunch(n, seed=seed)


def _refpts(ring, refs):
    if refs == 0:
        return np.zeros(0, dtype=np.uint32)
    n = len(_ring(ring))
    return (np.arange(refs) * (n // refs)).astype(np.uint32)


def _jobs(case):
    """(ring name, particles, turns) of every job of a batch."""
    k = case["jobs"]
    return [("variant%d" % (2 + i), max(1, case["n"] // 2 + i * case["n"] // k),
             max(1, case["turns"] - i % 3)) for i in range(k)]


def _diff_inputs(case, seed, strengths):
    """Particles 1e-6 around the orbit, strengths within 1e-4 of the design,
    a cotangent of the final coordinates."""
    rng = np.random.default_rng(seed)
    r0 = 1e-6 * rng.standard_normal((case["n"], 6))
    k = np.array([float(_ring("fodo")[p.index].PolynomB[p.order]) for p in strengths])
    k = k * (1.0 + 1e-4 * rng.standard_normal(k.size))
    return r0, k, rng.standard_normal((case["n"], 6))


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case)
    if kind == "track":
        s["line"] = _ring(case["ring"])
        s["refpts"] = _refpts(case["ring"], case["refs"])
        s["r0"] = _particles(case["ring"], case["beam"], case["n"], seed)
    elif kind == "resident":
        n = case["n"]
        s["eng"] = Engine.get(0)
        s["lid"] = s["eng"].upload(_table(case["ring"])[0])
        s["r0"] = torch.from_numpy(
            np.ascontiguousarray(_particles(case["ring"], "bunch", n, seed).T)).cuda()
        s["r"] = torch.empty_like(s["r0"])
        s["loss"] = [torch.empty(sh, dtype=dt, device="cuda") for sh, dt in (
            ((n,), torch.uint8), ((n,), torch.int32), ((n,), torch.int32),
            ((n, 6), torch.float64))]
        s["stream"] = torch.cuda.Stream()
        torch.cuda.synchronize()
    elif kind == "batch":
        jobs = _jobs(case)
        s["bt"] = BatchTracker([_ring(j[0]) for j in jobs],
                               [rings.da_grid(j[1], seed + i) for i, j in enumerate(jobs)],
                               [j[2] for j in jobs], tune=False)
    else:
        ring = _ring("fodo")
        strengths = diff.multipole_strengths(ring)
        s["tr"] = (diff.AdjointTracker if kind == "adjoint" else diff.TangentTracker)(ring,
                                                                                    strengths)
        s["r0"], s["k"], s["g"] = (torch.from_numpy(a).cuda()
                                   for a in _diff_inputs(case, seed, strengths))
        if kind == "adjoint":
            s["r0"].requires_grad_()
            s["k"].requires_grad_()
    return s


def run(state):
    s = state
    kind = s["kind"]
    if kind == "track":
        r = s["r0"].copy(order="F")
        res = gpupass(s["line"], r, s["turns"], s["refpts"], losses=s["losses"],
                      reuse=s["reuse"], mode=s["mode"])
        rout, loss = res if s["losses"] else (res, None)
        return {"r": r, "rout": rout, "loss": loss}
    if kind == "resident":
        with torch.cuda.stream(s["stream"]):
            s["r"].copy_(s["r0"])
            for t in s["loss"]:
                t.zero_()
            s["eng"].track_device(s["lid"], s["r"].data_ptr(), s["n"], s["turns"],
                                  losses=tuple(t.data_ptr() for t in s["loss"]),
                                  mode=s["mode"], stream=s["stream"].cuda_stream)
        return {"r": s["r"], "loss": s["loss"]}
    if kind == "batch":
        s["bt"].reset()
        s["bt"].run()
        return s["bt"].results()
    if kind == "tangent":
        r, jac, grad, lost = s["tr"].track(s["r0"], s["k"], s["turns"])
        return {"r": r, "jac": jac, "grad": grad, "lost": lost}
    r = diff.track(s["tr"], s["r0"], s["k"], s["turns"])
    g_r0, g_k = torch.autograd.grad(r, (s["r0"], s["k"]), s["g"])
    return {"r": r, "g_r0": g_r0, "g_k": g_k}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        jobs = _jobs(case)
        return {"bytes": sum(n * 153 + _table(j)[0].words.nbytes for j, n, _ in jobs),
                "flops": sum(n * t * _table(j)[1] for j, n, t in jobs)}
    n, turns = case["n"], case["turns"]
    cl, fpt = _table(case.get("ring", "fodo"))
    size, ops = 96 * n + cl.words.nbytes, n * turns * fpt
    if kind == "tangent":      # the value and seven derivative directions
        return {"bytes": size + 8 * n * (36 + 6 * 128), "flops": 8 * ops}
    if kind == "adjoint":      # forward, and a reverse sweep of twice its work
        return {"bytes": size + 96 * n, "flops": 3 * ops}
    if kind == "resident" or case["losses"]:
        size += 57 * n
    return {"bytes": size + 48 * n * turns * case.get("refs", 0), "flops": ops}


# ---------------------------------------------------------------------------
# the same results in plain 64-bit numpy or torch
# ---------------------------------------------------------------------------
_C0 = 2.99792458e8
_CBRT2 = 2.0 ** (1.0 / 3.0)
_D1, _D2 = 0.5 / (2.0 - _CBRT2), 0.5 - 0.5 / (2.0 - _CBRT2)     # Forest-Ruth
_K1, _K2 = 1.0 / (2.0 - _CBRT2), 1.0 - 2.0 / (2.0 - _CBRT2)
_R_E = 2.8179403205e-15


def _field(a, b, x, y):
    re, im = b[-1], a[-1]
    for bn, an in zip(b[-2::-1], a[-2::-1]):
        re, im = re * x - im * y + bn, im * x + re * y + an
    return re, im


def _element(xp, el, r, turn, t0, gamma, energy, strength=None):
    """One element of a ring on the coordinates (x, px, y, py, d, ct);
    ``strength`` = (order, value) replaces a PolynomB coefficient."""
    x, px, y, py, d, ct = r
    pm = el.PassMethod
    if pm in ("IdentityPass", "AperturePass"):
        if pm == "AperturePass":
            lo, hi, bo, to = (float(v) for v in el.Limits)
            out = (x < lo) | (x > hi) | (y < bo) | (y > to)
            ct = xp.where(out, math.inf, ct)
        return x, px, y, py, d, ct
    if pm == "RFCavityPass":
        f = float(el.Frequency)
        slip = round(f * t0) / f - t0
        phase = 2.0 * math.pi * f * ((ct - float(getattr(el, "TimeLag", 0.0))) / _C0 -
                                     slip * turn)
        return x, px, y, py, d - float(el.Voltage) / energy * xp.sin(phase), ct
    length = float(el.Length)
    if pm == "DriftPass":
        pn = 1.0 / (1.0 + d)
        return (x + length * pn * px, px, y + length * pn * py, py, d,
                ct + 0.5 * length * pn * pn * (px * px + py * py))
    rad = pm.endswith("RadPass")
    bend = pm.startswith("Bnd")
    pn = 1.0 / (1.0 + d)
    if getattr(el, "T1", None) is not None:
        x, px, y, py, d, ct = (c + float(t) if float(t) else c
                               for c, t in zip((x, px, y, py, d, ct), el.T1))
    if getattr(el, "R1", None) is not None:
        x, px, y, py = _rotate(el.R1, x, px, y, py)
    irho = float(el.BendingAngle) / length if bend else 0.0
    if bend:
        e = irho * math.tan(float(el.EntranceAngle))
        px, py = px + x * e, py - y * e
    mo = int(el.MaxOrder)
    a, b = [float(v) for v in el.PolynomA[:mo + 1]], [float(v) for v in el.PolynomB[:mo + 1]]
    if strength is not None:
        b[strength[0]] = strength[1]
    step = length / int(el.NumIntSteps)
    stages = ((_D1, _K1), (_D2, _K2), (_D2, _K1), (_D1, None))
    radc = 2.0 / 3.0 * _R_E * gamma ** 3
    for _ in range(int(el.NumIntSteps)):
        for cd, ck in stages:
            nl = step * cd * pn
            x, y = x + nl * px, y + nl * py
            ct = ct + 0.5 * nl * pn * (px * px + py * py)
            if ck is None:
                continue
            lk = step * ck
            re, im = _field(a, b, x, y)
            dpx = -lk * (re - (d - x * irho) * irho) if bend else -lk * re
            if rad:
                xa, ya = px * pn, py * pn
                h = 1.0 + x * irho
                by = re + irho
                s = xa * xa + ya * ya
                b2 = ((by * by + im * im) * h * h + (im * ya - by * xa) ** 2) / (h * h + s)
                d = d - radc * b2 * (h + 0.5 * s) / (pn * pn) * lk
                pn = 1.0 / (1.0 + d)
                px, py = xa * (1.0 + d), ya * (1.0 + d)
            px, py = px + dpx, py + lk * im
            if bend:
                ct = ct + lk * irho * x
    if bend:
        e = irho * math.tan(float(el.ExitAngle))
        px, py = px + x * e, py - y * e
    if getattr(el, "R2", None) is not None:
        x, px, y, py = _rotate(el.R2, x, px, y, py)
    if getattr(el, "T2", None) is not None:
        x, px, y, py, d, ct = (c + float(t) if float(t) else c
                               for c, t in zip((x, px, y, py, d, ct), el.T2))
    return x, px, y, py, d, ct


def _rotate(m, x, px, y, py):
    c, s = float(m[0, 0]), float(m[0, 2])
    return c * x + s * y, c * px + s * py, c * y - s * x, c * py - s * px


def _constants(line):
    t0 = 0.0
    for el in line:
        t0 += float(getattr(el, "Length", 0.0))
    return t0 / _C0, float(line.energy) / float(line.particle.rest_energy), float(line.energy)


def _lost_now(xp, r):
    bad = ~xp.isfinite(r[5])
    for c in r[:5]:
        bad = bad | ~(abs(c) <= 1.0)
    return bad


def _exact_track(line, r0, turns, refpts):
    """Final coordinates and snapshots of the rows of ``r0`` (N, 6)."""
    small = r0.shape[0] < 3000
    xp = np if small else torch
    r = tuple(np.ascontiguousarray(r0[:, k]) if small else torch.from_numpy(r0[:, k].copy()).cuda()
              for k in range(6))
    lost = r[0] != r[0]
    const = _constants(line)
    refs, snaps = set(int(i) for i in refpts), []

    def rows(r):
        m = xp.stack(r)
        m = xp.where(lost[None, :], 0.0, m)
        m[0] = xp.where(lost, math.nan, m[0])
        return m

    with np.errstate(all="ignore"):
        for turn in range(turns):
            for i, el in enumerate(line):
                if i in refs:
                    snaps.append(rows(r))
                r = _element(xp, el, r, turn, *const)
                lost = lost | _lost_now(xp, r)
        return rows(r), snaps


def _gradients(line, strengths, r0, k, turns, cotangents):
    """Per-particle products with the ``cotangents`` ((C, N, 6)): the final
    coordinates, d/d r0 (C, N, 6) and d/d K (C, P, N), by reverse-mode
    differentiation of the plain tracking above, a few elements at a time."""
    const = _constants(line)
    at = {p.index: (q, p.order) for q, p in enumerate(strengths)}
    n = r0.shape[0]
    r = tuple(torch.from_numpy(np.ascontiguousarray(r0[:, j])).cuda() for j in range(6))
    kk = torch.from_numpy(k).cuda()[:, None].expand(-1, n)
    # particles times elements recorded at a time
    span = max(1, min(24, 6000000 // max(n, 1)))
    chunks = [(t, i, min(i + span, len(line))) for t in range(turns)
              for i in range(0, len(line), span)]

    def through(r, turn, lo, hi, ks):
        for i in range(lo, hi):
            q = at.get(i)
            r = _element(torch, line[i], r, turn, *const,
                         strength=None if q is None else (q[1], ks[q[0]]))
        return r

    entry = []
    with torch.no_grad():
        for c in chunks:
            entry.append(r)
            r = through(r, *c, kk)
    final = torch.stack(r, 1)
    lam = torch.from_numpy(cotangents).cuda()
    g_k = torch.zeros((lam.shape[0], len(strengths), n), dtype=torch.float64, device="cuda")
    for c, r in zip(chunks[::-1], entry[::-1]):
        r = tuple(v.detach().requires_grad_() for v in r)
        here = [at[i][0] for i in range(c[1], c[2]) if i in at]
        ks = {q: kk[q].clone().requires_grad_() for q in here}
        out = torch.stack(through(r, *c, ks), 1)
        g = torch.autograd.grad(out, r + tuple(ks[q] for q in here), lam, is_grads_batched=True,
                                allow_unused=True, materialize_grads=True)
        lam = torch.stack(g[:6], 2)
        for q, v in zip(here, g[6:]):
            g_k[:, q] += v
    return final, lam, g_k


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return None
    n, turns = case["n"], case["turns"]
    fpt = _table(case.get("ring", "fodo"))[1]
    if kind in ("track", "resident"):
        if fpt * turns * (1e-6 + 1e-9 * n if n < 3000 else 6e-6 + 1e-11 * n) > 20.0:
            return None
        line, refs = _ring(case["ring"]), case.get("refs", 0)
        refpts = _refpts(case["ring"], refs)
        r0 = _particles(case["ring"], case.get("beam", "bunch"), n, seed).T
        r, snaps = _exact_track(line, np.ascontiguousarray(r0), turns, refpts)
        if not isinstance(r, np.ndarray):
            r, snaps = r.cpu().numpy(), [s.cpu().numpy() for s in snaps]
        if kind == "resident":
            return {"r": np.ascontiguousarray(r.T), "loss": None}
        rout = np.zeros((6, n, refs, turns))
        for j, s in enumerate(snaps):
            rout[:, :, j % refs, j // refs] = s
        loss = None
        if case["losses"]:
            loss = {"islost": None, "turn": None, "elem": None, "coord": None}
        return {"r": r, "rout": rout, "loss": loss}
    if fpt * turns * (2e-5 + 2e-10 * n * (6 if kind == "tangent" else 1)) > 25.0:
        return None
    strengths = diff.multipole_strengths(_ring("fodo"))
    r0, k, g = _diff_inputs(case, seed, strengths)
    if kind == "adjoint":
        r, g_r0, g_k = _gradients(_ring("fodo"), strengths, r0, k, turns, g[None])
        return {"r": r, "g_r0": g_r0[0], "g_k": g_k[0].sum(1)}
    rows = np.broadcast_to(np.eye(6)[:, None, :], (6, n, 6)).copy()
    r, jac, grad = _gradients(_ring("fodo"), strengths, r0, k, turns, rows)
    return {"r": r, "jac": jac.permute(1, 0, 2).contiguous(),
            "grad": grad.permute(1, 0, 2).contiguous(), "lost": None}
