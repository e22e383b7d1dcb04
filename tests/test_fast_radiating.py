"""The fast kernels' radiating magnets inside and outside the range of their
reciprocals' series (angles above 3 mrad, a path factor further than 2^-9 from
one, large losses): within the fast arithmetic's 1e-13 of each coordinate's
scale over one element, on either side and with both in one warp."""
import numpy as np
import pytest

from at_b200 import elements as E
from at_b200.lattice import compile_lattice
from oracle import oracle

from conftest import ELECTRON_REST, scale_rel_diff


def _particles(kind):
    rng = np.random.default_rng(3)
    r = rng.standard_normal((6, 200)) * np.array([1e-3, 1e-4, 1e-3, 1e-4, 1e-3, 1e-3])[:, None]
    if kind == "wide":
        r[0] = rng.uniform(-0.08, 0.08, 200)          # path factors, strong fields
        r[1] = rng.uniform(-0.02, 0.02, 200)          # angles
        r[4] = rng.uniform(-0.1, 0.1, 200)
    elif kind == "mixed":
        r[1, ::7] = rng.uniform(-0.02, 0.02, r[1, ::7].size)
    return np.asfortranarray(r)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["bunch", "mixed", "wide"])
@pytest.mark.parametrize("bend", [False, True])
@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_fast_radiating_magnet(kind, bend, order):
    from at_b200.engine import Engine
    b = [0.0, 0.3, -4.0, 50.0, 100.0][:order + 1]
    kw = dict(BendingAngle=0.06, EntranceAngle=0.02, ExitAngle=0.03) if bend else {}
    el = E.Element("M", 0.5, PassMethod="%sMPoleSymplectic4RadPass" % ("Bnd" if bend else "Str"),
                   PolynomA=[0.0] * (order + 1), PolynomB=b, MaxOrder=order, NumIntSteps=4, **kw)
    r0 = _particles(kind)
    ro = r0.copy(order="F")
    oracle.track([el], ro, 1, energy=6e9, rest_energy=ELECTRON_REST, element=True, t0=0.0)
    rg = r0.copy(order="F")
    eng = Engine.get(0)
    lid = eng.upload(compile_lattice([el], 6e9, ELECTRON_REST, t0=0.0))
    try:
        eng.track(lid, rg, 1, element=True, mode="fast")
    finally:
        eng.free(lid)
    assert scale_rel_diff(rg, ro) <= 1e-13
