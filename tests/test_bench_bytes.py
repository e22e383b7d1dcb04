"""The bytes that the bench declares for a drop-in call: a call that loses
nothing copies the coordinates and the loss flags back, not the whole map."""
import importlib.util
import os

import numpy as np

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_bytes_copied_back():
    spec = importlib.util.spec_from_file_location("bench", os.path.join(REPO, "bench.py"))
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    lost = np.zeros(1000, dtype=bool)
    assert bench.d2h_bytes(1000, {"islost": lost}) == 49000
    lost[7] = True
    assert bench.d2h_bytes(1000, {"islost": lost}) == 105000
