"""The adjoint sweep of strong magnets (focusing phases up to 6 rad a magnet,
sextupoles and octupoles with large gradients at the particle, bends among
them, plain and misaligned) against the tangent kernel, which never walks
backwards.

Both propagate the same derivatives, so dL/dr0 agrees to the roundings of a few
hundred operations on terms of the size |J|^T |g|: 1e-13 of it.  (With the
coordinates found by undoing such a magnet dL/d delta is off by 2e-12 of it at
6 rad.)  The tangent kernel takes a strength's derivatives through J^-1, with an
error of cond(J) roundings of |dr/dK| |g|: ten times that is allowed there."""
import numpy as np
import pytest

from at_b200 import diff, rings
from at_b200 import elements as E

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SHIFT = dict(T1=[1e-5, 0, -2e-5, 0, 0, 0], T2=[-1e-5, 0, 2e-5, 0, 0, 0],
             R1=rings._rot(0.05), R2=rings._rot(-0.05))
MAGNETS = {
    "quad": lambda **k: E.Quadrupole("Q", 2.0, -9.0, **k),
    "quad_many_steps": lambda **k: E.Quadrupole("Q", 2.0, 9.0, NumIntSteps=37, **k),
    "quad_at_the_line": lambda **k: E.Quadrupole("Q", 1.0, 4.04, **k),
    "sextupole": lambda **k: E.Sextupole("S", 1.0, 4000.0, **k),
    "octupole": lambda **k: E.Octupole("O", 1.0, [], [0.0, 0.0, 0.0, 4e6], **k),
    "skew": lambda **k: E.Multipole("M", 1.5, [0.0, 5.0, 300.0], [0.0, 4.0, 500.0], NumIntSteps=10, **k),
    "bend": lambda **k: E.Dipole("B", 2.0, 0.3, -8.0, EntranceAngle=0.1, ExitAngle=0.2, **k),
    "bend_sext": lambda **k: E.Dipole("B", 1.0, 0.3, PolynomB=[0.0, 3.0, 900.0], MaxOrder=2,
                                      PolynomA=[0.0] * 3, **k),
}


@pytest.mark.parametrize("place", ["plain", "misaligned"])
@pytest.mark.parametrize("name", sorted(MAGNETS))
def test_strong_magnet_equals_the_tangent(name, place):
    el = MAGNETS[name](**(SHIFT if place == "misaligned" else {}))
    line = E.Lattice([E.Drift("D", 0.1), el, E.Drift("D", 0.2), E.Quadrupole("Q", 0.3, 1.0)],
                     energy=3e9, particle="electron", name="strong")
    order = len(np.trim_zeros(np.asarray(el.PolynomB), "b")) - 1
    ps = [(1, order), (3, 1)]
    adj, tan = diff.AdjointTracker(line, ps), diff.TangentTracker(line, ps)
    rng = np.random.default_rng(1)
    r0 = rng.standard_normal((300, 6)) * np.array([2e-4, 2e-5, 1e-4, 1e-5, 1e-3, 1e-3])
    r0, g = (torch.from_numpy(a).cuda() for a in (r0, rng.standard_normal((300, 6))))
    r, jac, grad, lost = tan.track(r0, None, 1)
    assert not lost.any()
    for kw in (dict(), dict(store_elements=True)):
        ra, lost, state = adj.forward(r0, None, 1, **kw)
        g_r0, g_k = adj.backward(state, g)
        assert torch.equal(ra, r) and not lost.any()
        size = torch.einsum("nij,ni->nj", jac.abs(), g.abs())
        want = torch.einsum("nij,ni->nj", jac, g)
        assert ((g_r0 - want).abs() / size).max() <= 1e-13
        size = torch.einsum("pin,ni->p", grad.abs(), g.abs())
        want = torch.einsum("pin,ni->p", grad, g)
        assert ((g_k - want).abs() / size).max() <= 10 * 2.0 ** -53 * torch.linalg.cond(jac).max()
    adj.close()
    tan.close()
