"""The exact kernels' reciprocals (at_b200/csrc/atb_rn.h) over the ranges of
ordinary rings: on the CPU against the hardware's division, on the GPU bending
and straight magnets from 1 to 50 GeV against the oracle, bit for bit.
"""
import ctypes as C
import math
import os
import subprocess

import numpy as np
import pytest

from at_b200 import elements as E
from at_b200.lattice import compile_lattice
from oracle import oracle

from conftest import ELECTRON_REST, ROOT

SOURCE = r"""
#include <stdbool.h>
#include "atb_rn.h"
void near_(long n, const double* d, double* q) { for (long i = 0; i < n; ++i) q[i] = rn_rcp_near(d[i]); }
void from_(long n, const double* o, const double* s, double* q, int* ok) { for (long i = 0; i < n; ++i)
  { double e; q[i] = rn_rcp_from(o[i], s[i], &e); ok[i] = rn_below(e, ATB_RN_SEED_HI); } }
void wide_(long n, const double* o, const double* s, double* q, int* ok) { for (long i = 0; i < n; ++i)
  { double e; q[i] = rn_rcp_from_wide(o[i], s[i], &e); ok[i] = rn_below(e, rn_seed_wide_hi(10)); } }
void factor_(long n, const double* a, const double* o, const double* p, double* q) { for (long i = 0; i < n; ++i)
  { double p2 = p[i] * p[i]; q[i] = rn_div(a[i], p2, rn_rcp_step(p2, o[i] * o[i])); } }
void div_(long n, const double* a, const double* b, const double* y, double* q)
{ for (long i = 0; i < n; ++i) q[i] = rn_div(a[i], b[i], y[i]); }
void ordinary_(long n, const double* a, double* q) { for (long i = 0; i < n; ++i) q[i] = rn_ordinary(a[i]); }
void ranges_(long n, const double* a, double* q) { for (long i = 0; i < n; ++i)
  q[i] = rn_opd_constant(a[i]) + 2 * rn_opd_fits(a[i]); }
"""


@pytest.fixture(scope="module")
def rn(tmp_path_factory):
    d = tmp_path_factory.mktemp("rn")
    src, so = d / "rn.c", d / "rn.so"
    src.write_text(SOURCE)
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-o", str(so), str(src),
                    "-I", os.path.join(ROOT, "at_b200", "csrc"), "-lm"], check=True)
    lib = C.CDLL(str(so))

    def call(name, *arrays, flags=False):
        n = arrays[0].size
        args = [np.ascontiguousarray(a, dtype=np.float64) for a in arrays]
        out, ok = np.empty(n), np.empty(n, dtype=np.int32)
        ptrs = [a.ctypes.data_as(C.c_void_p) for a in (*args, out)]
        if flags:
            ptrs.append(ok.ctypes.data_as(C.c_void_p))
        getattr(lib, name)(C.c_long(n), *ptrs)
        return (out, ok.astype(bool)) if flags else out
    return call


N = 1_000_000
#: significands at which a reciprocal's last rounding is hardest
EDGES = np.concatenate([1.0 + np.arange(64) * 2.0 ** -52, 2.0 - (1 + np.arange(64)) * 2.0 ** -52])


def test_reciprocals_of_any_size(rn):
    rng = np.random.default_rng(0)
    d = rng.uniform(1.0, 2.0, N) * np.ldexp(1.0, rng.integers(-900, 900, N))
    d = np.concatenate([d, 1.0 + rng.uniform(-0.3, 0.3, N), EDGES, 0.5 * EDGES, EDGES * 2.0 ** 300,
                        1.0 + np.ldexp(rng.uniform(-1, 1, N), rng.integers(-53, -1, N))])
    np.testing.assert_array_equal(rn("near_", d), 1.0 / d)


@pytest.mark.parametrize("name,bits", [("from_", 18), ("wide_", 14)])
def test_reciprocals_from_a_neighbour(rn, name, bits):
    rng = np.random.default_rng(bits)
    before = np.concatenate([rng.uniform(0.7072, 1.4141, N), 1.0 + rng.integers(-64, 65, N) * 2.0 ** -53])
    e = rng.uniform(-1, 1, before.size) * np.ldexp(1.0, -rng.integers(bits, 54, before.size))
    o = before * (1.0 + e)
    o[:1000] = 1.0 - 2.0 ** -53
    before[:1000] = 1.0 - np.arange(1000) * 2.0 ** -53
    q, ok = rn(name, o, 1.0 / before, flags=True)
    assert ok.mean() > 0.97
    np.testing.assert_array_equal(q[ok], 1.0 / o[ok])
    assert not rn(name, np.array([1.0, np.inf, np.nan]), np.array([1.0 + 2.0 ** -13, 1.0, 1.0]),
                  flags=True)[1].any()


def test_quotients_over_the_momentum_range(rn):
    rng = np.random.default_rng(3)
    o = rng.uniform(0.7072, 1.4141, N)
    a = rng.uniform(-2.0, 2.0, N)
    p = 1.0 / o
    np.testing.assert_array_equal(rn("factor_", a, o, p), a / (p * p))
    np.testing.assert_array_equal(rn("div_", a, p, o), a / p)
    o = np.concatenate([rng.uniform(0.5, 2.0, N), EDGES, 0.5 * EDGES])
    a = rng.uniform(1.0, 2.0, o.size) * np.ldexp(1.0, rng.integers(-850, 850, o.size))
    np.testing.assert_array_equal(rn("div_", a, 2.0 * o, 0.5 / o), a / (2.0 * o))


def test_accepted_operands(rn):
    a = np.array([0.0, -0.0, 1.0, -1.0, 2.0 ** -480, np.nextafter(2.0 ** -480, 0.0), 2.0 ** -1074,
                  -2.0 ** -1043, 2.0 ** -1000, 2.0 ** 399, 2.0 ** 400, np.inf, np.nan])
    assert rn("ordinary_", a).tolist() == [1, 1, 1, 1, 1, 0, 0, 0, 0, 1, 0, 0, 0]
    a = np.array([0.5, np.nextafter(0.5, 0), 97 / 128, np.nextafter(97 / 128, 0), 1.0,
                  np.nextafter(1.25, 0), 1.25, np.nextafter(2, 0), 2.0, -1.0, np.nan])
    assert rn("ranges_", a).tolist() == [1, 0, 3, 1, 3, 3, 1, 1, 0, 0, 0]


#: light-source dipoles: energy, length, number in the ring
RINGS = [(3e9, 0.6, 224), (3e9, 1.0, 64), (3e9, 1.4, 32), (6e9, 1.0, 64), (6e9, 2.3, 64), (8e9, 2.8, 88)]


def _kick_loss(energy, length, angle, steps):
    """The largest relative energy loss of one kick in a dipole's own field:
    (2/3) r_e gamma^3 (angle/length)^2 times the longest kick, 1.7024 steps."""
    gamma = energy / ELECTRON_REST
    return 2.0 / 3.0 * 2.8179403205e-15 * gamma ** 3 * (angle / length) ** 2 * 1.7024 * length / steps


@pytest.mark.parametrize("energy,length,number", RINGS)
def test_ordinary_dipoles_are_inside_the_range(rn, energy, length, number):
    """Ten steps a dipole, and particles in three times the dipole's field."""
    loss = _kick_loss(energy, length, 2 * math.pi / number, 10)
    o = np.array([1.0 - 9.0 * loss])
    q, ok = rn("wide_", o, np.array([1.0]), flags=True)
    assert ok.all() and q[0] == 1.0 / o[0]


# -- on the GPU -----------------------------------------------------------------

def _particles():
    rng = np.random.default_rng(5)
    r = rng.standard_normal((6, 256)) * np.array([1e-3, 1e-4, 1e-3, 1e-4, 1e-3, 1e-3])[:, None]
    r[:, :16] = 0.0
    r[4, :16] = np.linspace(-8, 7, 16) * 2.0 ** -53         # 1 + delta next to one
    r[0, 16:80] = np.linspace(-0.3, 0.3, 64)                # far from the axis
    r[1, 80:112] = np.linspace(-0.3, 0.3, 32)               # steep
    r[4, 112:160] = np.linspace(-0.55, 0.9, 48)             # off momentum
    return np.asfortranarray(r)


def _track(el, r0, energy, ppt=1):
    from at_b200.engine import Engine
    eng = Engine.get(0)
    lid = eng.upload(compile_lattice([el], energy, ELECTRON_REST, t0=0.0))
    r = r0.copy(order="F")
    eng.set_launch(particles_per_thread=ppt)
    try:
        eng.track(lid, r, 1, element=True, mode="exact")
    finally:
        eng.set_launch(particles_per_thread=1)
        eng.free(lid)
    return r


@pytest.mark.gpu
@pytest.mark.parametrize("steps", [1, 10, 257])
@pytest.mark.parametrize("energy", [1e9, 3e9, 6e9, 8e9, 20e9, 50e9])
def test_radiating_bends_equal_the_oracle(energy, steps):
    """At 3 GeV and ten steps the 96 ordinary particles' kicks are inside the
    bound (2^-14) by the formula, at 50 GeV outside."""
    el = E.Dipole("B", 0.6, 0.05, 0.5, EntranceAngle=0.02, ExitAngle=0.03, NumIntSteps=steps,
                  PassMethod="BndMPoleSymplectic4RadPass")
    loss = _kick_loss(energy, 0.6, 0.05, steps)
    if steps == 10:
        assert (loss < 2.0 ** -15) == (energy < 10e9)
    r0 = _particles()
    ro = r0.copy(order="F")
    oracle.track([el], ro, 1, energy=energy, rest_energy=ELECTRON_REST, element=True, t0=0.0)
    np.testing.assert_array_equal(_track(el, r0, energy), ro)


def _dense(seed):
    return np.eye(6) + 1e-3 * np.random.default_rng(seed).standard_normal((6, 6))


@pytest.mark.gpu
@pytest.mark.parametrize("ppt", [1, 2])
@pytest.mark.parametrize("form", [dict(), dict(T1=[1e-5, 0, 0, 0, 1e-4, 0]),
                                  dict(R1=_dense(1), R2=_dense(2)),
                                  dict(T1=[0, 0, 0, 0, 1e-4, 0], R1=_dense(1))])
@pytest.mark.parametrize("method", ["StrMPoleSymplectic4Pass", "StrMPoleSymplectic4RadPass",
                                    "BndMPoleSymplectic4Pass", "BndMPoleSymplectic4RadPass"])
def test_entrances_that_change_the_momentum(method, form, ppt):
    kw = {}
    if method.startswith("Bnd"):                  # attributes that a bend has to have
        kw = dict(BendingAngle=0.05, EntranceAngle=0.02, ExitAngle=0.03)
    el = E.Element("M", 0.4, PassMethod=method, PolynomA=[0.0, 0.0], PolynomB=[0.0, 1.3], MaxOrder=1,
                   NumIntSteps=4, **kw, **form)
    r0 = _particles()
    if ppt == 2:                                  # enough particles for full tiles of two each
        r0 = np.asfortranarray(np.tile(r0, (1, 500)))
    ro = r0.copy(order="F")
    oracle.track([el], ro, 1, energy=3e9, rest_energy=ELECTRON_REST, element=True, t0=0.0)
    np.testing.assert_array_equal(_track(el, r0, 3e9, ppt), ro)


@pytest.mark.gpu
@pytest.mark.parametrize("steps", [4096, 4097])
def test_magnets_of_many_steps(steps):
    """From 4097 steps on the table leaves the flag of these quotients unset."""
    el = E.Quadrupole("Q", 0.4, 1.3, NumIntSteps=steps, PassMethod="StrMPoleSymplectic4RadPass")
    r0 = _particles()[:, :64].copy(order="F")
    ro = r0.copy(order="F")
    oracle.track([el], ro, 1, energy=3e9, rest_energy=ELECTRON_REST, element=True, t0=0.0)
    np.testing.assert_array_equal(_track(el, r0, 3e9), ro)
