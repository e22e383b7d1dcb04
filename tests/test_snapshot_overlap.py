"""Snapshots that come back while the next turns are tracked: the same as one
launch's, for chunks of turns of every kind (a short last one, a partial first
turn, losses, statistics), and a loss map that holds zeros where nothing was
lost."""
import numpy as np
import pytest

from at_b200 import rings
from at_b200.engine import Engine
from at_b200.lattice import compile_lattice

pytestmark = pytest.mark.gpu


def _track(eng, lid, r0, turns, refs, **kw):
    r = r0.copy(order="F")
    rout, loss, stats = eng.track(lid, r, turns, refpts=refs, **kw)
    return r, rout, loss, stats


@pytest.mark.parametrize("turns", [2, 4, 5, 9])
@pytest.mark.parametrize("start", [0, 100])
def test_overlapped_snapshots_equal_separate_turns(turns, start):
    ring = rings.fodo_ring()
    eng = Engine.get(0)
    lid = eng.upload(compile_lattice(ring, ring.energy, ring.particle.rest_energy))
    refs = np.array([0, 7, 101, 250, 385], dtype=np.uint32)
    # (a first turn that starts past a point waits for it in vain and takes no
    # snapshot at all, as the reference's walk does: its points come after)
    refs = refs[refs >= start]
    n = 40009 if start == 0 else 70009            # 10 MB a turn: piped from two turns on
    r0 = rings.gaussian(n, [5e-3, 1e-4, 3e-3, 1e-4, 1e-2, 1e-3], seed=turns)
    try:
        r, rout, loss, stats = _track(eng, lid, r0, turns, refs, losses=True, stats=True,
                                      start_elem=start)
        one = r0.copy(order="F")
        lost = np.zeros(n, dtype=bool)
        for t in range(turns):
            _, part, l, st = (one,) + eng.track(lid, one, 1, turn0=t, refpts=refs, losses=True,
                                                stats=True, start_elem=start if t == 0 else 0)
            keep = ~lost                          # a call forgets who was lost before
            np.testing.assert_array_equal(rout[:, keep, :, t], part[:, keep, :, 0])
            lost |= np.isnan(one[0])
            assert stats[0][t] == (~lost).sum()
        np.testing.assert_array_equal(r, one)
        np.testing.assert_array_equal(loss["islost"], lost)
        assert lost.any() and (loss["turn"][~lost] == 0).all()
    finally:
        eng.free(lid)


def test_loss_map_without_losses_is_zero():
    ring = rings.fodo_ring()
    eng = Engine.get(0)
    lid = eng.upload(compile_lattice(ring, ring.energy, ring.particle.rest_energy))
    try:
        for n, sigma in ((1, 1e-6), (5000, 1e-6), (5000, 0.3)):
            r0 = rings.gaussian(n, [sigma] * 6, seed=1)
            _, _, loss, _ = _track(eng, lid, r0, 1, None, losses=True)
            if sigma < 1e-3:
                for k in ("islost", "turn", "elem", "coord"):
                    assert not loss[k].any()
            else:
                assert loss["islost"].any() and np.any(loss["coord"][:, loss["islost"]] != 0)
                assert not loss["coord"][:, ~loss["islost"]].any()
    finally:
        eng.free(lid)
