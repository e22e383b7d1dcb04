"""The error of the hand-written tangent kernel against differences taken in
binary128, beside that of the one on dual numbers: no larger.

One turn of the FODO ring, whose 64 equal bends round alike.  The differences
are central ones at two steps, extrapolated: their own error is below 1e-20 of
an entry.  Both kernels track the same 128 particles, so the ratio of the errors'
root mean squares varies by a few per cent; a tenth is allowed."""
import numpy as np
import pytest

from at_b200 import diff, rings
from at_b200 import elements as E
from oracle import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _jacobian(line, r0):
    out = np.zeros((r0.shape[0], 6, 6))
    for j in range(6):
        est = []
        for h in (2.0 ** -26, 2.0 ** -27):
            a, b = (r0.T.copy(order="F") for _ in range(2))
            a[j] += h
            b[j] -= h
            p, m = (oracle.track_quad(line, v, 1, energy=line.energy,
                                      rest_energy=line.particle.rest_energy) for v in (a, b))
            est.append(((p[0] - m[0]) + (p[1] - m[1])) / (a[j] - b[j]))
        out[:, :, j] = ((4.0 * est[1] - est[0]) / 3.0).T
    return out


def test_no_further_from_binary128_than_dual_numbers():
    line = rings.fodo_ring()
    r0 = 1e-6 * np.random.default_rng(0).standard_normal((128, 6))
    want = _jacobian(line, r0)
    scale = np.abs(want).max(axis=0)
    # one radiating element of no length leads to the dual-number kernel
    extra = E.Multipole("none", 0.0, [0.0], [0.0], MaxOrder=0, NumIntSteps=1,
                        PassMethod="StrMPoleSymplectic4RadPass")
    dual = E.Lattice([*line, extra], energy=line.energy, particle=line.particle, name="dual")
    error = []
    for ring in (line, dual):
        tr = diff.TangentTracker(ring)
        jac = tr.track(torch.from_numpy(r0).cuda())[1].cpu().numpy()
        tr.close()
        e = (jac - want)[:, scale > 0] / scale[scale > 0]
        error.append(np.sqrt((e ** 2).mean()))
    assert error[1] < 1e-12
    assert error[0] <= 1.1 * error[1], error
