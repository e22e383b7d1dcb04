"""The exact kernels' quotients (at_b200/csrc/atb_rn.h) against IEEE division.

On the CPU the same header is compiled for the host and compared with the
hardware's division over the operands the kernels accept; on the GPU single
magnets are tracked at the edges of the accepted ranges and beyond them (where
the plain expressions take over) and must equal the oracle bit for bit.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from at_b200 import elements as E
from at_b200.lattice import compile_lattice
from oracle import oracle

from conftest import ELECTRON_REST, ROOT

SOURCE = r"""
#include "atb_rn.h"
void div_(long n, const double* a, const double* b, const double* y, double* q)
{ for (long i = 0; i < n; ++i) q[i] = rn_div(a[i], b[i], y[i]); }
void step_(long n, const double* d, const double* y, double* q)
{ for (long i = 0; i < n; ++i) q[i] = rn_rcp_step(d[i], y[i]); }
void from_(long n, const double* o, const double* s, double* q, int* ok)
{ for (long i = 0; i < n; ++i) { double e; q[i] = rn_rcp_from(o[i], s[i], &e);
    ok[i] = rn_below(e, ATB_RN_SEED_HI) && rn_opd_fits(o[i]) && !rn_below_one(o[i]); } }
void nearer_(long n, const double* d, double* q, int* ok)
{ for (long i = 0; i < n; ++i) { q[i] = rn_rcp_nearer(d[i]); ok[i] = rn_nearer_fits(d[i]); } }
void near_(long n, const double* d, double* q, int* ok)
{ for (long i = 0; i < n; ++i) { q[i] = rn_rcp_near(d[i]); ok[i] = rn_near_fits(d[i]); } }
#define TEST_FN(name, f) void name(long n, const double* a, int* ok) \
{ for (long i = 0; i < n; ++i) ok[i] = f; }
TEST_FN(square_, rn_square_fits(a[i]))
TEST_FN(tiny_, rn_not_tiny(a[i]))
TEST_FN(denormal_, rn_denormal(a[i]))
TEST_FN(x_, rn_coords_fit(a[i], 1.0, 0.0, -1.0))
TEST_FN(px_, rn_coords_fit(-0.0, a[i], 1.0, 1.0))
TEST_FN(y_, rn_coords_fit(1.0, 0.0, a[i], 0.0))
TEST_FN(py_, rn_coords_fit(0.0, 0.0, -1.0, a[i]))
"""


@pytest.fixture(scope="module")
def rn(tmp_path_factory):
    d = tmp_path_factory.mktemp("rn")
    src, so = d / "rn.c", d / "rn.so"
    src.write_text("#include <stdbool.h>\n" + SOURCE)
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-o", str(so), str(src),
                    "-I", os.path.join(ROOT, "at_b200", "csrc"), "-lm"], check=True)
    lib = C.CDLL(str(so))

    def call(name, *arrays, flags=False, test=False):
        n = arrays[0].size
        args = [np.ascontiguousarray(a, dtype=np.float64) for a in arrays]
        out, ok = np.empty(n), np.empty(n, dtype=np.int32)
        ptrs = [a.ctypes.data_as(C.c_void_p) for a in args]
        if not test:
            ptrs.append(out.ctypes.data_as(C.c_void_p))
        if flags:
            ptrs.append(ok.ctypes.data_as(C.c_void_p))
        getattr(lib, name)(C.c_long(n), *ptrs)
        if test:
            return ok.astype(bool)
        return (out, ok.astype(bool)) if flags else out
    return call


def _numerators(rng, n):
    """Significands anywhere, next to one and next to two; wide exponents."""
    a = rng.uniform(1.0, 2.0, n)
    k = rng.integers(0, 64, n) * 2.0 ** -52
    pick = rng.integers(0, 3, n)
    a = np.where(pick == 1, 1.0 + k, np.where(pick == 2, 2.0 - 2.0 ** -52 - k, a))
    return a * np.ldexp(1.0, rng.integers(-850, 850, n)) * rng.choice([-1.0, 1.0], n)


def _near_one(rng, n, half):
    """Numbers within ``half`` of one, many of them a few ulps from it."""
    close = 1.0 + rng.integers(-64, 65, n) * 2.0 ** -53
    any_ = 1.0 + half * rng.uniform(-1, 1, n) * np.ldexp(1.0, -rng.integers(0, 50, n))
    return np.where(rng.random(n) < 0.3, close, any_)


def test_quotients_equal_ieee_division(rn):
    rng = np.random.default_rng(0)
    n = 2_000_000
    o = _near_one(rng, n, 0.125)
    o = o[(o >= 0.875) & (o < 1.125)]
    a = _numerators(rng, o.size)
    p = 1.0 / o
    np.testing.assert_array_equal(rn("div_", a, 2.0 * o, 0.5 * p), a / (2.0 * o))
    keep = o != 1.0 - 2.0 ** -53
    o, a, p = o[keep], a[keep], p[keep]
    np.testing.assert_array_equal(rn("div_", a, p, o), a / p)
    num = _near_one(rng, o.size, 0.01)
    p2 = p * p
    np.testing.assert_array_equal(rn("div_", num, p2, rn("step_", p2, o * o)), num / p2)


def test_zero_numerators_keep_their_sign(rn):
    for z in (0.0, -0.0):
        for o in (0.9, 1.0, 1.1):
            q = rn("div_", np.array([z]), np.array([1.0 / o]), np.array([o]))
            assert q[0] == 0.0 and np.signbit(q[0]) == np.signbit(z)


def test_reciprocals_equal_ieee_division(rn):
    rng = np.random.default_rng(1)
    n = 2_000_000
    d = _near_one(rng, n, 2.0 ** -8)
    q, ok = rn("near_", d, flags=True)
    assert ok.mean() > 0.9
    np.testing.assert_array_equal(q[ok], 1.0 / d[ok])
    d = 1.0 + rng.uniform(0, 1, n) * np.ldexp(1.0, -rng.integers(9, 53, n))
    q, ok = rn("nearer_", d, flags=True)
    assert ok.mean() > 0.9
    np.testing.assert_array_equal(q[ok], 1.0 / d[ok])
    seed = 1.0 / _near_one(rng, n, 0.125)
    o = (1.0 / seed) * (1.0 + rng.uniform(-1, 1, n) * np.ldexp(1.0, -rng.integers(19, 54, n)))
    q, ok = rn("from_", o, seed, flags=True)
    assert 0.5 < ok.mean() < 1.0
    np.testing.assert_array_equal(q[ok], 1.0 / o[ok])


def test_accepted_operands(rn):
    """Each test's bound; zeros pass, nothing else that is tiny does except
    denormals with a zero high word, which have a test of their own."""
    for name, low in (("square_", -860), ("tiny_", -480), ("x_", -400), ("px_", -400),
                      ("y_", -400), ("py_", -400)):
        lo = 2.0 ** low
        a = np.array([0.0, 1.0, lo, np.nextafter(lo, 0.0), 2.0 ** -1040, 2.0 ** -1074])
        ok = [True, True, True, False, False, True]
        if name != "square_":                       # the others take either sign
            a, ok = np.concatenate((a, -a)), ok + ok
        assert rn(name, a, flags=True, test=True).tolist() == ok, name
    a = np.array([0.0, -0.0, 5e-324, -5e-324, 2.0 ** -1043, 2.0 ** -1042, 1.0, np.inf])
    assert rn("denormal_", a, flags=True, test=True).tolist() == [
        False, False, True, True, True, False, False, False]


def test_table_flag_of_the_shared_quotients():
    """ATB_F_RN: lengths within range and at most 4096 steps."""
    from at_b200 import table as T
    for length, ns, ok in ((0.4, 10, True), (0.0, 3, True), (-0.4, 4096, True), (0.4, 4097, False),
                           (2.0 ** 45, 1, False), (2.0 ** -45, 1, False), (0.4, 0, False)):
        el = E.Multipole("M", length, [0.0, 0.0], [0.0, 1.0], NumIntSteps=ns)
        cl = compile_lattice([el], 3e9, ELECTRON_REST)
        assert bool(cl.info[0].flags & T.ATB_F_RN) == ok, (length, ns)


# -- on the GPU -----------------------------------------------------------------

def _edge_particles():
    """Coordinates inside the accepted ranges, at their edges and outside."""
    rng = np.random.default_rng(2)
    base = rng.standard_normal((6, 160)) * np.array([1e-3, 1e-4, 1e-3, 1e-4, 1e-2, 1e-3])[:, None]
    base[:, :8] = 0.0                                        # on the axis
    base[2:4, 8:24] = 0.0                                    # flat, either plane
    base[0:2, 24:40] = 0.0
    base[4, 40:72] = np.linspace(-0.13, 0.13, 32)            # 1 + delta around 7/8 and 9/8
    base[4, 72:80] = [2.0 ** -53, -2.0 ** -53, -2.0 ** -54, 2.0 ** -52, 1e-300, -1e-16, 0.0, -0.0]
    base[3, 80:96] = np.ldexp(1.0, -np.linspace(390, 1074, 16).astype(int))   # tiny angles
    base[1, 88:96] = 0.0
    base[0, 96:112] = np.linspace(0.05, 0.9, 16)             # far from the axis
    base[1, 112:128] = np.linspace(0.01, 0.5, 16)            # steep
    base[4, 128:132] = [-1.0, -0.999, 0.9, 1.5]
    base[0, 132:136] = [1e10, -1e150, 1e200, np.inf]
    base[3, 136:140] = [1e10, 1e160, -np.inf, np.nan]
    base[5, 140:142] = [np.inf, np.nan]
    return np.asfortranarray(base)


POLY = {"order0": ([0.0], [0.02]), "quad": ([0.0, 0.0], [0.0, 1.3]),
        "sext": ([0.0, 0.0, 0.0], [0.0, 0.1, -60.0]),
        "octu": ([0.0] * 4, [0.0, 0.0, 0.0, 900.0]), "deca": ([0.0] * 5, [0.0, 0.0, 0.0, 0.0, 1e4]),
        "skew": ([1e-3, 0.2], [0.0, 1.3]), "minus_zero": ([-0.0, -0.0], [-0.0, 0.7])}


@pytest.mark.gpu
@pytest.mark.parametrize("poly", sorted(POLY))
@pytest.mark.parametrize("method", ["StrMPoleSymplectic4Pass", "StrMPoleSymplectic4RadPass",
                                    "BndMPoleSymplectic4Pass", "BndMPoleSymplectic4RadPass"])
@pytest.mark.parametrize("ppt", [1, 2])
def test_magnets_at_the_edges_equal_the_oracle(method, poly, ppt):
    from at_b200.engine import Engine
    a, b = POLY[poly]
    kw = {}
    if method.startswith("Bnd"):
        kw = dict(BendingAngle=0.05, EntranceAngle=0.02, ExitAngle=0.03)
    el = E.Element("M", 0.4, PassMethod=method, PolynomA=a, PolynomB=b, MaxOrder=len(b) - 1,
                   NumIntSteps=3, T1=[1e-5, 0, 0, 0, 1e-4 if poly == "skew" else 0, 0], **kw)
    r0 = _edge_particles()
    if ppt == 2:                                  # enough particles for full tiles of two each
        r0 = np.asfortranarray(np.tile(r0, (1, 800)))
    ro = r0.copy(order="F")
    oracle.track([el], ro, 1, energy=6e9, rest_energy=ELECTRON_REST, element=True, t0=0.0)
    rg = r0.copy(order="F")
    eng = Engine.get(0)
    lid = eng.upload(compile_lattice([el], 6e9, ELECTRON_REST, t0=0.0))
    eng.set_launch(particles_per_thread=ppt)
    try:
        eng.track(lid, rg, 1, element=True, mode="exact")
    finally:
        eng.set_launch(particles_per_thread=1)
        eng.free(lid)
    np.testing.assert_array_equal(rg, ro)
