"""The radial stage and the constraint kernel at every edge of their tables (the
smallest and largest column of each compiled length, odd and even), on planes whose
level rows are multiples of 16 bytes in every field, in pairs only, or in none, and
on one with several tiles per block.  Bounds are those of the oracle comparisons in
test_gpu_parity.py and of its mixed-precision steps."""
import numpy as np
import pytest

from test_gpu_parity import random_fields, relmax

pytestmark = pytest.mark.gpu

# 63, 60, 54 sites: odd, a multiple of 4, of 2 only
CASES = [(nz, *p) for i, nz in enumerate([4, 5, 8, 9, 12, 13, 16, 17, 18, 21, 22, 25, 26, 32, 33])
         for p in [[(7, 9), (10, 6), (6, 9)][i % 3]]] + [(21, 101, 99), (9, 100, 98), (33, 99, 98)]


@pytest.mark.parametrize("nz,nx,ny", CASES)
def test_rhs(hqt, oracle, dev, nz, nx, ny):
    to_d, from_d = dev
    Lx, Ly = 0.5 * nx, 0.45 * ny
    Z = random_fields(nx, ny, nz, seed=nz)
    op = oracle.build_operators(nx, ny, nz, Lx, Ly)
    F1, F2, F3, F4 = oracle.rhs(op, *Z)
    with hqt.Simulation(nx, ny, nz, Lx=Lx, Ly=Ly) as sim:
        g1, g2b, g3, g4 = sim.rhs_device(*[to_d(z) for z in Z])
    for got, want in ((from_d(g1), F1), (from_d(g3), F3), (from_d(g4), F4),
                      (g2b.cpu().numpy().T, F2[:, :, -1])):
        assert relmax(got, want) < 1e-11


@pytest.mark.parametrize("nz,nx,ny", CASES)
def test_step(hqt, oracle, dev, nz, nx, ny):
    """Also: a repeat gives the same bits, and mixed precision the same fields."""
    L = 0.5 * nx
    prof = hqt.seed.stationary_profile(6.0, -2 * np.pi * 7 / 20)
    state = list(hqt.seed.init_driven(nx, ny, nz, prof, noise="complex", amplitude=1e-2, seed=nz))
    op = oracle.build_operators(nx, ny, nz, L)
    want, _ = oracle.rk4_step(op, oracle.OracleState(*[a.copy() for a in state]), 0.005, 6.0,
                              prof.vy, False)
    kw = dict(Lx=L, Ly=L, mu=6.0, vy=prof.vy, dt=0.005, remove_winding=False)
    with hqt.Simulation(nx, ny, nz, **kw) as sim:
        got, _ = sim.step(*state, nsteps=1)
        again, _ = sim.step(*state, nsteps=1)
    with hqt.Simulation(nx, ny, nz, precision="mixed", **kw) as sim:
        mixed, _ = sim.step(*state, nsteps=1)
    scale = np.linalg.norm(want.Z2.ravel())
    for g, a, m, r in zip(got, again, mixed, (want.Z1, want.Z2, want.Z3, want.Z4, want.rhoi)):
        assert np.array_equal(g, a)
        n = max(np.linalg.norm(r.ravel()), scale)
        assert np.linalg.norm((g - r).ravel()) < 1e-12 * n
        assert np.linalg.norm((m - r).ravel()) < 1e-8 * n
