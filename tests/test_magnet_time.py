"""A magnet takes the same time wherever its particles are and whatever it
radiates: one integration loop covers large angles, particles far from the axis
and the energy losses of 6 and 8 GeV dipoles, where a second loop beside it
would take more than twice the time.  The same instructions run, so the times
differ by the timer's noise; a quarter is allowed.
"""
import math

import numpy as np
import pytest

from at_b200 import elements as E
from at_b200.elements import Lattice
from at_b200.lattice import compile_lattice

from conftest import ELECTRON_REST

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

N = 4096
RAD = "%sMPoleSymplectic4RadPass"


def _quad():
    return E.Quadrupole("Q", 0.02, 1e-3, PassMethod=RAD % "Str")


def _bend(length=0.05, rho=7.0):
    return E.Dipole("B", length, length / rho, PassMethod=RAD % "Bnd")


#: name: (element, energy in eV, coordinate, its size at the reference, its size outside)
CASES = {
    "off momentum, no radiation": (E.Quadrupole("Q", 0.2, 1e-3), 3e9, 4, 1e-4, 3e-1),
    "angles": (_quad(), 3e9, 1, 1e-4, 3e-2),
    "far from a bend's axis": (_bend(), 3e9, 0, 1e-5, 4e-2),
    "a compact bend": (_bend(rho=1.0), 1e9, 0, 1e-5, 2e-2),
}
#: dipoles by energy: length, angle (ten steps each)
DIPOLES = {3e9: (1.4, 2 * math.pi / 32), 6e9: (2.3, 2 * math.pi / 64), 8e9: (2.8, 2 * math.pi / 88)}


def _time(el, energy, coord, size, mode):
    from at_b200.engine import Engine
    eng = Engine.get(0)
    line = Lattice([el] * 40, energy=energy, particle="electron")
    lid = eng.upload(compile_lattice(line, energy, ELECTRON_REST))
    r0 = 1e-7 * np.random.default_rng(0).standard_normal((N, 6))
    r0[:, coord] = size * np.linspace(-1.0, 1.0, N)
    r0 = torch.from_numpy(r0).cuda()
    st, best = torch.cuda.Stream(), math.inf
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        for _ in range(8):
            r = r0.clone()
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            eng.track_device(lid, r.data_ptr(), N, 1, mode=mode, stream=st.cuda_stream)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
    eng.free(lid)
    assert not torch.isnan(r).any()
    return best


@pytest.mark.parametrize("mode", ["exact", "fast"])
@pytest.mark.parametrize("case", sorted(CASES))
def test_time_does_not_depend_on_the_coordinates(case, mode):
    el, energy, coord, near, far = CASES[case]
    assert _time(el, energy, coord, far, mode) <= 1.25 * _time(el, energy, coord, near, mode)


@pytest.mark.parametrize("mode", ["exact", "fast"])
@pytest.mark.parametrize("energy", sorted(DIPOLES))
def test_time_does_not_depend_on_the_energy_loss(energy, mode):
    length, angle = DIPOLES[energy]
    el = E.Dipole("B", length, angle, PassMethod=RAD % "Bnd")
    assert _time(el, energy, 0, 1e-5, mode) <= 1.25 * _time(el, 1e9, 0, 1e-5, mode)


@pytest.mark.parametrize("mode", ["exact", "fast"])
def test_time_does_not_depend_on_what_an_entrance_rotation_mixes(mode):
    """A dense rotation that changes delta takes a division more a magnet than
    one that leaves it."""
    keep = np.eye(6) + 1e-9 * np.random.default_rng(0).standard_normal((6, 6))
    mixes = keep.copy()
    keep[4] = np.eye(6)[4]
    times = [_time(E.Quadrupole("Q", 0.2, 1e-3, R1=r), 3e9, 0, 1e-6, mode) for r in (mixes, keep)]
    assert times[0] <= 1.25 * times[1]
