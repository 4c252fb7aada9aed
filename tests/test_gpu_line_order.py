"""A right-hand side with runtime line plans gives the same bits each time: lengths along
y whose butterfly counts are no multiple of the block size (the blocks' warps then drift
apart between barriers), on enough slices to fill the device."""
import numpy as np
import pytest

from test_gpu_parity import random_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(64, 100), (66, 180), (64, 250), (48, 384), (21, 1001)])
def test_rhs_repeats_its_bits(hqt, dev, nx, ny):
    to_d, _ = dev
    nz = 33
    Z = [to_d(z) for z in random_fields(nx, ny, nz, seed=ny)]
    with hqt.Simulation(nx, ny, nz, Lx=0.5 * nx, Ly=0.45 * ny) as sim:
        first = [f.clone() for f in sim.rhs_device(*Z)]
        for _ in range(200):
            for f, want in zip(sim.rhs_device(*Z), first):
                assert bool((f == want).all())
    assert all(np.isfinite(f.abs().sum().item()) for f in first)
