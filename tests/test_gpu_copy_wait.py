"""A radial kernel that waits in vain for a copy gives up, waits for its copies in flight
and ends with a fault, which the call reports; the context stays usable.  The wait is
made to run out by allowing it no poll at all."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

POLLS = 1 << 20  # the kernels' own limit


def set_polls(hqt, sim, polls):
    fn = hqt._lib.load().hqt_set_copy_polls
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int]
    assert fn(sim._ctx, polls) == 0


def run_state(hqt, nx, ny, nz):
    prof = hqt.seed.stationary_profile(6.0, -2 * np.pi * 7 / 20)
    return hqt.seed.init_driven(nx, ny, nz, prof, noise="complex", amplitude=1e-2, seed=nz)


# level rows of 16-byte multiples and others, one tile and several a block
@pytest.mark.parametrize("nx,ny,nz,precision", [
    (12, 14, 8, "fp64"), (33, 33, 21, "fp64"), (33, 33, 21, "mixed"), (256, 250, 21, "fp64"),
    (48, 100, 33, "fp64"), (301, 301, 33, "mixed")])
def test_a_lost_copy_is_an_error_and_the_context_goes_on(hqt, cuda, nx, ny, nz, precision):
    state = run_state(hqt, nx, ny, nz)
    kw = dict(Lx=0.5 * nx, Ly=0.5 * ny, mu=6.0, vy=-2.0, dt=0.005, precision=precision)
    with hqt.Simulation(nx, ny, nz, **kw) as sim:
        want, _ = sim.step(*state, nsteps=2)
        for _ in range(3):
            set_polls(hqt, sim, 0)
            with pytest.raises(hqt.HQTError, match="copies did not arrive") as e:
                sim.step(*state, nsteps=2)
            assert e.value.code == hqt._lib.HQT_ECUDA
            set_polls(hqt, sim, POLLS)
            got, info = sim.step(*state, nsteps=2)
            assert info.steps_done == 2
            assert all(np.array_equal(g, w) for g, w in zip(got, want))


def test_a_right_hand_side_after_a_fault(hqt, dev):
    """A fault is reported by the call it happened in, not by the next one."""
    to_d, _ = dev
    state = run_state(hqt, 33, 33, 21)
    Z = [to_d(a) for a in state[:4]]
    with hqt.Simulation(33, 33, 21, Lx=16.5, mu=6.0, vy=-2.0) as sim:
        want = [f.clone() for f in sim.rhs_device(*Z)]
        for call in (lambda: sim.rhs_device(*Z), lambda: sim.step(*state, nsteps=1)):
            set_polls(hqt, sim, 0)
            with pytest.raises(hqt.HQTError, match="copies did not arrive"):
                call()
            set_polls(hqt, sim, POLLS)
            for f, w in zip(sim.rhs_device(*Z), want):
                assert bool((f == w).all())


def test_an_ensemble_reports_a_lost_copy(hqt, dev):
    to_d, from_d = dev
    grids = (24, 33)
    states = [run_state(hqt, n, n, 12) for n in grids]
    sims = [hqt.Simulation(n, n, 12, Lx=0.5 * n, mu=6.0, vy=-2.0, dt=0.005) for n in grids]

    def run():
        now = [[to_d(a) for a in s] for s in states]
        with hqt.Ensemble(sims) as ens:
            ens.step_device(now, nsteps=2)
        return [[from_d(t) for t in s] for s in now]

    want = run()
    set_polls(hqt, sims[1], 0)
    with pytest.raises(hqt.HQTError, match="copies did not arrive"):
        run()
    set_polls(hqt, sims[1], POLLS)
    for g, w in zip(run(), want):
        assert all(np.array_equal(a, b) for a, b in zip(g, w))
