"""Derivative calls and prepared batches of one engine from several streams:
the strength maps, scratch and launch lists they share belong to one call at a
time, so every call gets the result it gets alone.

The final coordinates, Jacobians and cotangents are the same operations in the
same order, hence equal bits; the strengths' gradients are sums over particles
in an order that varies from run to run, hence equal to the roundings of a sum
of n terms, n 2^-53 times the sum of their sizes.
"""
import numpy as np
import pytest

from at_b200 import diff, rings
from at_b200.batch import BatchTracker

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _sets(trackers, sizes):
    out = []
    for i, (tr, n) in enumerate(zip(trackers, sizes)):
        rng = np.random.default_rng(i)
        r0 = torch.from_numpy(1e-6 * rng.standard_normal((n, 6))).cuda()
        g = torch.from_numpy(rng.standard_normal((n, 6))).cuda()
        out.append((tr, r0, tr.k0 * (1.0 + 1e-3 * i), g))
    torch.cuda.synchronize()
    return out


def _adjoint(tr, r0, k, g, stride):
    r, lost, state = tr.forward(r0, k, 3, stride=stride)
    return (r, *tr.backward(state, g))


def _alone_and_together(run, sets):
    alone = []
    for s in sets:
        alone.append(run(*s))
        torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in sets]
    for _ in range(3):
        together = []
        for s, st in zip(sets, streams):
            with torch.cuda.stream(st):
                together.append(run(*s))
        torch.cuda.synchronize()
    return alone, together


def _trackers(cls):
    """Three trackers of one ring with different strengths."""
    ring = rings.fodo_ring()
    ps = diff.multipole_strengths(ring)
    return [cls(ring, p) for p in (ps, ps[::-1][:40], ps[3:90])]


@pytest.mark.parametrize("stride", [1, 2])
def test_adjoint_trackers_on_streams_of_their_own(stride):
    sets = _sets(_trackers(diff.AdjointTracker), (9001, 2001, 5003))
    alone, together = _alone_and_together(lambda *s: _adjoint(*s, stride), sets)
    for (tr, r0, k, g), a, b in zip(sets, alone, together):
        assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
        n = r0.shape[0]
        # |dL/dK| of one particle times the particles, over all strengths
        size = n * a[2].abs().max()
        assert (a[2] - b[2]).abs().max() <= n * 2.0 ** -53 * size
        tr.close()


def test_tangent_trackers_on_streams_of_their_own():
    sets = _sets(_trackers(diff.TangentTracker), (3001, 301, 1003))
    alone, together = _alone_and_together(lambda tr, r0, k, g: tr.track(r0, k, 1), sets)
    for s, a, b in zip(sets, alone, together):
        for u, v in zip(a, b):
            assert torch.equal(u, v)
        s[0].close()


@pytest.mark.parametrize("graph", [False, True])
def test_one_batch_launched_on_two_streams(graph):
    """The second launch goes on from the first's particles."""
    ring = rings.fodo_ring()
    bt = BatchTracker([ring, ring], [rings.gaussian(n, seed=n) for n in (30001, 701)], [4, 7],
                      tune=False, graph=graph)
    ends = []
    for wait in (True, False):
        bt.reset()
        for _ in range(2):
            bt.eng.batch_launch(bt.bid, stream=torch.cuda.Stream().cuda_stream)
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        ends.append([r for r, _ in bt.results()])
    for a, b in zip(*ends):
        np.testing.assert_array_equal(a, b)
    bt.close()
