"""Launches of one engine from several streams: each waits for the last before
the engine's launch lists are replaced, so every set gets its own result."""
import numpy as np
import pytest

from at_b200 import rings
from at_b200.engine import Engine
from at_b200.lattice import compile_lattice

torch = pytest.importorskip("torch")


@pytest.mark.gpu
def test_two_streams_without_waiting_between():
    ring = rings.fodo_ring()
    eng = Engine.get(0)
    lid = eng.upload(compile_lattice(ring, ring.energy, ring.particle.rest_energy))
    sizes, turns = (40000, 9001, 70001), (6, 3, 4)
    starts = [torch.from_numpy(np.ascontiguousarray(rings.gaussian(n, seed=i).T)).cuda()
              for i, n in enumerate(sizes)]
    alone = []
    for r0, t in zip(starts, turns):
        st = torch.cuda.Stream()
        st.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(st):
            r = r0.clone()
            eng.track_device(lid, r.data_ptr(), r.shape[0], t, stream=st.cuda_stream)
        torch.cuda.synchronize()
        alone.append(r)
    streams = [torch.cuda.Stream() for _ in starts]
    together = [r0.clone() for r0 in starts]
    torch.cuda.synchronize()
    for _ in range(3):
        for r, r0, t, st in zip(together, starts, turns, streams):
            with torch.cuda.stream(st):
                r.copy_(r0)
                eng.track_device(lid, r.data_ptr(), r.shape[0], t, stream=st.cuda_stream)
    torch.cuda.synchronize()
    for a, b in zip(together, alone):
        torch.testing.assert_close(a, b, rtol=0, atol=0, equal_nan=True)
    eng.free(lid)
