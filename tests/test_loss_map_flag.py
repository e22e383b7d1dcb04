"""atb_track's loss map as a C caller sees it: without ATB_FLAG_ZEROED every
array is written whatever it held; with it, the arrays beyond the flags are left
alone when nothing was lost and written when something was."""
import numpy as np
import pytest

from at_b200 import _lib, rings
from at_b200._lib import check, lib, ptr
from at_b200.engine import Engine
from at_b200.lattice import compile_lattice

pytestmark = pytest.mark.gpu
FILL = {"islost": 0xA5, "turn": 0xDEADBEEF, "elem": 0xDEADBEEF, "coord": -7.25}


def _track(eng, lid, r, flags):
    n = r.shape[1]
    out = {"islost": np.full(n, FILL["islost"], dtype=np.uint8),
           "turn": np.full(n, FILL["turn"], dtype=np.uint32),
           "elem": np.full(n, FILL["elem"], dtype=np.uint32),
           "coord": np.full((6, n), FILL["coord"], order="F")}
    with eng.lock:
        check(lib().atb_track(eng.h, int(lid), ptr(r), n, 2, 0, 0, eng.nelem[lid], None, 0, None, 1,
                              ptr(out["islost"]), ptr(out["turn"]), ptr(out["elem"]),
                              ptr(out["coord"]), None, None, _lib.MODE_EXACT, flags))
    return out


@pytest.mark.parametrize("lost", [(), (5, 300)])
@pytest.mark.parametrize("flags", [0, _lib.FLAG_ZEROED])
def test_loss_map_into_arrays_that_hold_something(flags, lost):
    ring = rings.fodo_ring()
    eng = Engine.get(0)
    lid = eng.upload(compile_lattice(ring, ring.energy, ring.particle.rest_energy))
    r0 = rings.gaussian(1000, seed=1)
    r0[1, list(lost)] = 0.9
    _, want, _ = eng.track(lid, r0.copy(order="F"), 2, losses=True, mode="exact")
    assert want["islost"].sum() == len(lost)
    got = _track(eng, lid, r0.copy(order="F"), flags)
    eng.free(lid)
    np.testing.assert_array_equal(got["islost"], want["islost"].astype(np.uint8))
    for k in ("turn", "elem", "coord"):
        if flags and not lost:
            assert (got[k] == np.array(FILL[k], dtype=got[k].dtype)).all()
        else:
            np.testing.assert_array_equal(got[k], want[k])
