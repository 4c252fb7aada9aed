"""What a context costs before its first call."""
import time

import pytest

pytestmark = pytest.mark.gpu


def test_a_small_context_is_made_quickly(hqt, cuda):
    """One device allocation and the kernels of its own lengths: 0.8 ms (6.8 with one
    allocation an array and the kernels of every length)."""
    best = 1.0
    for _ in range(20):
        t = time.perf_counter()
        sim = hqt.Simulation(64, 64, 21)
        best = min(best, time.perf_counter() - t)
        sim.close()
    assert best < 3e-3
