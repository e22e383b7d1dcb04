"""Thin elements and drifts with apertures, in each form that the element loop
treats by itself (plain, misaligned, with field scaling, with apertures), in the
exact kernel bit for bit against the oracle, and their cost beside a drift's."""
import math

import numpy as np
import pytest

from at_b200 import elements as E
from at_b200.elements import Lattice
from at_b200.lattice import compile_lattice
from oracle import oracle

from conftest import ELECTRON_REST

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SHIFT = dict(T1=[1e-4, 0, -2e-4, 0, 0, 0], T2=[-1e-4, 0, 2e-4, 0, 0, 0])
RECT = dict(RApertures=[-0.01, 0.01, -0.005, 0.005])
ELLIP = dict(EApertures=[0.01, 0.005])
FORMS = {
    "marker": lambda: E.Marker("M"), "marker_shift": lambda: E.Marker("M", **SHIFT),
    "marker_rect": lambda: E.Marker("M", **RECT),
    "corrector": lambda: E.Corrector("C", 0.0, [1e-4, -2e-4]),
    "corrector_shift": lambda: E.Corrector("C", 0.0, [1e-4, -2e-4], **SHIFT),
    "corrector_scaled": lambda: E.Corrector("C", 0.0, [1e-4, -2e-4], FieldScaling=1.01),
    "corrector_thick": lambda: E.Corrector("C", 0.1, [1e-4, -2e-4]),
    "thin0": lambda: E.ThinMultipole("T", [1e-4], [2e-4]),
    "thin2": lambda: E.ThinMultipole("T", [1e-4, 0.02, 0.3], [2e-4, -0.1, 5.0]),
    "thin5": lambda: E.ThinMultipole("T", [0.0] * 6, [0.0, 0.1, 0.0, 0.0, 0.0, 1e6]),
    "thin_bend": lambda: E.ThinMultipole("T", [0.0, 0.0], [0.0, 0.1], BendingAngle=np.array([0.01, 0.02])),
    "thin_shift": lambda: E.ThinMultipole("T", [0.0, 0.0], [0.0, 0.1], **SHIFT),
    "thin_scaled": lambda: E.ThinMultipole("T", [0.0, 0.0], [0.0, 0.1], FieldScaling=1.01),
    "drift_rect": lambda: E.Drift("D", 0.7, **RECT), "drift_ellip": lambda: E.Drift("D", 0.7, **ELLIP),
    "drift_both": lambda: E.Drift("D", 0.7, **RECT, **ELLIP),
    "drift_shift_rect": lambda: E.Drift("D", 0.7, **SHIFT, **RECT),
    "aperture": lambda: E.Aperture("A", [-0.01, 0.01, -0.005, 0.005]),
    "quad_both": lambda: E.Quadrupole("Q", 0.3, 1.1, **RECT, **ELLIP),
    "bend_rect": lambda: E.Dipole("B", 0.3, 0.02, **RECT),
}


def _particles():
    """A bunch, particles on each aperture's edge and next to it, and particles
    that a coordinate loses."""
    rng = np.random.default_rng(7)
    r = rng.standard_normal((6, 128)) * np.array([4e-3, 5e-3, 2e-3, 2e-3, 1e-2, 1e-3])[:, None]
    edge = [0.01, -0.01, np.nextafter(0.01, 1), np.nextafter(-0.01, -1)]
    r[:, :8] = 0.0
    r[0, :4] = edge
    r[2, 4:8] = 0.5 * np.array(edge)
    r[0, 8], r[2, 9], r[5, 10], r[1, 11] = np.nan, np.inf, np.inf, 1.5
    return np.asfortranarray(r)


@pytest.mark.parametrize("form", sorted(FORMS))
def test_form_equals_the_oracle(form):
    from at_b200.engine import Engine
    line = [E.Drift("D", 0.1), FORMS[form](), E.Drift("D", 0.1)]
    cl = compile_lattice(line, 3e9, ELECTRON_REST, t0=0.0)
    assert all(i.error is None for i in cl.info)
    eng, r0 = Engine.get(0), _particles()
    lid = eng.upload(cl)
    ro, rg = r0.copy(order="F"), r0.copy(order="F")
    out = oracle.track(line, ro, 2, energy=3e9, rest_energy=ELECTRON_REST, t0=0.0, losses=True)
    _, loss, _ = eng.track(lid, rg, 2, losses=True, mode="exact")
    eng.free(lid)
    np.testing.assert_array_equal(rg, ro)
    lost = out[1]
    for k in ("islost", "turn", "elem", "coord"):
        np.testing.assert_array_equal(loss[k], lost[k])


def _time(el, mode):
    from at_b200.engine import Engine
    eng = Engine.get(0)
    lid = eng.upload(compile_lattice(Lattice([el] * 100, energy=3e9, particle="electron"), 3e9,
                                     ELECTRON_REST))
    r0 = torch.from_numpy(1e-7 * np.random.default_rng(0).standard_normal((2048, 6))).cuda()
    st, best = torch.cuda.Stream(), math.inf
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        for _ in range(8):
            r = r0.clone()
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            eng.track_device(lid, r.data_ptr(), r.shape[0], 8, mode=mode, stream=st.cuda_stream)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
    eng.free(lid)
    return best


@pytest.mark.parametrize("mode", ["exact", "fast"])
@pytest.mark.parametrize("form,drifts", [("marker", 1.6), ("corrector", 1.8), ("thin2", 2.9)])
def test_cost_beside_a_drift(form, drifts, mode):
    """Measured 1.2, 1.3 and 2.1 drifts (2.3, 2.7 and 3.4 when the whole particle
    went through a call)."""
    assert _time(FORMS[form](), mode) <= drifts * _time(E.Drift("D", 0.3), mode)
