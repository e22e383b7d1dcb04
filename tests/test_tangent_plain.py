"""The tangent kernel with hand-written element derivatives against the one on
dual numbers, over every element form it accepts.

The dual-number kernel is reached by one radiating element of no length, which
leaves the coordinates as they are up to a rounding.  Both propagate the same
derivatives through a few thousand operations, so they agree to about 1e3
roundings: 1e-12 of each derivative's scale over the particles.  A strength's
derivatives are J u with u from a linear solve, so they agree to 1e-11 of
sum_j |J_ij| |u_j|, the terms that cancel in the components a strength hardly
touches (delta moves only through the cavities).
"""
import numpy as np
import pytest

from at_b200 import diff, rings
from at_b200 import elements as E

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _tilt(t):
    r = np.eye(6)
    r[0, 0] = r[1, 1] = r[2, 2] = r[3, 3] = np.cos(t)
    r[0, 2] = r[1, 3] = np.sin(t)
    r[2, 0] = r[3, 1] = -np.sin(t)
    return r


def _dense(seed):
    return np.eye(6) + 1e-3 * np.random.default_rng(seed).standard_normal((6, 6))


def _lattice():
    shift = dict(T1=[1e-5, 0, -2e-5, 0, 0, 0], T2=[-1e-5, 0, 2e-5, 0, 0, 0])
    bend = dict(EntranceAngle=0.02, ExitAngle=0.03)
    line = [
        E.Drift("D", 0.3), E.Drift("DM", 0.2, R1=_tilt(1e-3), R2=_tilt(-1e-3), **shift),
        E.Quadrupole("Q", 0.5, 1.1), E.Quadrupole("QT", 0.4, -1.2, R1=_tilt(0.1), R2=_tilt(-0.1),
                                                  **shift),
        E.Sextupole("S", 0.2, 15.0), E.Octupole("O", 0.2, [], [0, 0, 0, 900.0]),
        E.Multipole("M5", 0.2, [0, 0, 0, 0, 0], [0, 0.1, 2.0, 0, 1e4]),
        E.Multipole("SK", 0.3, [1e-4, 0.2, 1.0], [0, 0.3, -4.0]),
        E.Multipole("C0", 0.3, [0.0], [1e-4], MaxOrder=0, NumIntSteps=1),
        E.Multipole("DP", 0.3, [0, 0], [0, 0.4], T1=[0, 0, 0, 0, 1e-4, 0]),
        E.Multipole("DR", 0.3, [0, 0], [0, 0.4], R1=_dense(1), R2=_dense(2)),
        E.Dipole("B", 1.0, 0.1, 0.3, **bend), E.Dipole("B0", 0.8, 0.05, 0.0, **bend),
        E.Dipole("BS", 0.8, 0.05, PolynomB=[0, -0.2, 3.0], PolynomA=[0, 0.01, 0], MaxOrder=2,
                 R1=_tilt(0.02), R2=_tilt(-0.02), **bend, **shift),
        E.ThinMultipole("T", [1e-5, 0.01, 0.3], [0, 0.02, -1.0], R2=_tilt(0.01)),
        E.Corrector("C", 0.0, [1e-6, -2e-6]), E.Marker("M", R1=_tilt(0.01), R2=_tilt(-0.01)),
        E.Aperture("A", [-0.1, 0.1, -0.1, 0.1]),
        E.RFCavity("RF", 0.0, 1e6, 3.3e8, 40, 3e9), E.RFCavity("RFL", 0.2, 5e5, 3.3e8, 40, 3e9),
    ]
    for k in (0, 1, 2):                       # edge methods with a fringe correction
        line.append(E.Dipole("BF", 0.7, 0.06, 0.1, FullGap=0.04, FringeInt1=0.5, FringeInt2=0.4,
                             FringeBendEntrance=k, FringeBendExit=2 - k, **bend))
    return E.Lattice(line, energy=3e9, particle="electron", name="forms")


def _with_dual(line):
    extra = E.Multipole("none", 0.0, [0.0], [0.0], MaxOrder=0, NumIntSteps=1,
                        PassMethod="StrMPoleSymplectic4RadPass")
    out = line.copy()
    out.append(extra)
    return E.Lattice(list(out), energy=line.energy, particle=line.particle, name=line.name)


def _strengths(line):
    want = {"Q": (1,), "QT": (1,), "S": (2,), "O": (3,), "M5": (4,), "SK": (2,), "B": (1,),
            "BS": (1,), "T": (2,), "DR": (1,)}
    return [(i, want[e.FamName][0]) for i, e in enumerate(line) if e.FamName in want]


def _close(a, b, tol, scale=None):
    a, b = a.cpu().numpy(), b.cpu().numpy()
    s = np.nanmax(np.abs(b), axis=0, keepdims=True) if scale is None else scale.cpu().numpy()
    s = np.where(s == 0, 1.0, s)
    assert np.array_equal(np.isnan(a), np.isnan(b))
    assert np.nanmax(np.abs(a - b) / s) <= tol


@pytest.mark.parametrize("n,turns", [(1, 1), (127, 1), (129, 2), (300, 0), (1000, 2)])
def test_every_form_equals_the_dual_numbers(n, turns):
    line = _lattice()
    ps = _strengths(line)
    a, b = diff.TangentTracker(line, ps), diff.TangentTracker(_with_dual(line), ps)
    rng = np.random.default_rng(n)
    r0 = rng.standard_normal((n, 6)) * np.array([1e-3, 1e-4, 1e-3, 1e-4, 1e-3, 1e-3])
    if n > 5:
        r0[2] = 0.0
        r0[3, 0] = 0.4                         # lost at the aperture
        r0[4, 4] = 0.12                        # beyond the range of the shared quotients
    r0 = torch.from_numpy(r0).cuda()
    k = a.k0 * (1 + 1e-3 * torch.arange(len(ps), device="cuda", dtype=torch.float64) / len(ps))
    ra, ja, ga, la = a.track(r0, k, turns)
    rb, jb, gb, lb = b.track(r0, k, turns)
    assert torch.equal(la, lb)
    if n > 5 and turns:
        assert la[3] and not la[[0, 2]].any()
    _close(ra, rb, 1e-13)
    _close(ja, jb, 1e-12 * max(turns, 1))
    g = torch.movedim(gb, 2, 0).transpose(1, 2)                   # (N, 6, P)
    jac = torch.where(lb[:, None, None], torch.eye(6, dtype=jb.dtype, device=jb.device), jb)
    u = torch.linalg.solve(jac, torch.nan_to_num(g))
    terms = torch.movedim((jac.abs() @ u.abs()).transpose(1, 2), 0, 2)
    _close(ga, gb, 1e-11, terms)
    a.close()
    b.close()


def test_values_equal_the_exact_kernel():
    from at_b200 import tracking
    line = _lattice()
    r0 = rings.gaussian(500, [1e-3, 1e-4, 1e-3, 1e-4, 1e-3, 1e-3], seed=4)
    tr = diff.TangentTracker(line, ())
    r, _, _, lost = tr.track(torch.from_numpy(np.ascontiguousarray(r0.T)).cuda(), None, 3)
    out = r0.copy(order="F")
    tracking.gpupass(line, out, 3, mode="exact")
    ok = ~lost.cpu().numpy()
    np.testing.assert_array_equal(r.cpu().numpy()[ok], out.T[ok])
    tr.close()
