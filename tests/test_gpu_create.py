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


def test_memory_per_site(hqt, cuda):
    """280 bytes a site, and 116 for the FP32 fields of a mixed step, apart from planes and
    tables."""
    nx, ny, nz = 512, 512, 25
    for precision, most in (("fp64", 280), ("mixed", 396)):
        cuda.cuda.synchronize()
        before = cuda.cuda.mem_get_info()[0]
        sim = hqt.Simulation(nx, ny, nz, precision=precision)
        used = before - cuda.cuda.mem_get_info()[0]
        sim.close()
        assert used < most * nx * ny * nz + (64 << 20)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny", [(40, 30), (301, 24), (64, 128)])
def test_host_and_device_runs_agree(hqt, dev, nx, ny, precision):
    """The state of a host run shares its place with stage fields: same bits as a run on
    the caller's arrays, with vortex counts and observables taken in between."""
    import numpy as np
    to_d, from_d = dev
    nz = 9
    prof = hqt.seed.stationary_profile(6.0, -2.0)
    state = hqt.seed.init_driven(nx, ny, nz, prof, noise="complex", amplitude=1e-2, seed=nx)
    for filt in (True, False):
        kw = dict(Lx=0.5 * nx, Ly=0.5 * ny, mu=6.0, vy=-2.0, dt=0.005, diag_every=2,
                  precision=precision, apply_filter=filt)
        with hqt.Simulation(nx, ny, nz, **kw) as sim:
            host, hi = sim.step(*state, nsteps=5, records=4)
            again, _ = sim.step(*state, nsteps=0)
        with hqt.Simulation(nx, ny, nz, **kw) as sim:
            t = [to_d(a) for a in state]
            di = sim.step_device(*t, nsteps=5, records=4)
        assert hi.steps_done == di.steps_done == 5
        assert len(hi.records) == 2 and np.array_equal(hi.records, di.records)
        assert all(np.array_equal(h, from_d(d)) for h, d in zip(host[:4], t))
        assert all(np.array_equal(a, b) for a, b in zip(again, state))
