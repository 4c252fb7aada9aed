"""The in-place line transforms (every length with prime factors up to 13) at
the plans where an index can go wrong: two passes of the smallest lines, every
radix as first and as last pass, equal large radices (11*11, 13*13), four
passes, odd lengths (no row swizzle), and lines that do not fill a block in
either direction.  Bounds are those of the oracle comparisons in
test_gpu_parity.py: the oracle's dense operators round more than a transform."""
import numpy as np
import pytest

from test_gpu_parity import random_fields, relmax, vortex_field

pytestmark = pytest.mark.gpu

# (nx, ny): x plan / y plan
GRIDS = [(4, 6), (9, 10), (12, 14), (22, 15), (26, 35), (121, 18), (20, 169), (143, 27),
         (98, 117), (250, 36), (45, 180), (33, 1001), (1001, 21), (24, 1024), (1000, 25),
         (768, 13 * 6), (50, 640), (128, 100), (100, 128), (66, 63)]


@pytest.mark.parametrize("nx,ny", GRIDS)
def test_rhs_and_filter(hqt, oracle, dev, nx, ny):
    to_d, from_d = dev
    nz = 5
    Lx, Ly = 0.5 * nx, 0.45 * ny
    Z1, Z2, Z3, Z4 = random_fields(nx, ny, nz, seed=nx + 3 * ny)
    op = oracle.build_operators(nx, ny, nz, Lx, Ly)
    F1, F2, F3, F4 = oracle.rhs(op, Z1, Z2, Z3, Z4)
    with hqt.Simulation(nx, ny, nz, Lx=Lx, Ly=Ly) as sim:
        g1, g2b, g3, g4 = sim.rhs_device(to_d(Z1), to_d(Z2), to_d(Z3), to_d(Z4))
        # an odd number of fields: the last has no imaginary partner
        x = np.stack([Z2, Z3, Z4])
        y = sim.filter_device(to_d(x.transpose(1, 2, 3, 0)).contiguous())
    for got, want in ((from_d(g1), F1), (from_d(g3), F3), (from_d(g4), F4),
                      (g2b.cpu().numpy().T, F2[:, :, -1])):
        assert relmax(got, want) < 1e-11
    want = np.stack([oracle.ff(f, op.mask) for f in x])
    assert relmax(from_d(y).transpose(3, 0, 1, 2), want) < 1e-12


@pytest.mark.parametrize("nx,ny", [(12, 14), (35, 26), (100, 128), (64, 98)])
def test_step_and_spectrum(hqt, oracle, dev, nx, ny):
    """Winding phase, real-pair derivatives and the forward y transform."""
    to_d, _ = dev
    nz, L = 7, 0.5 * nx
    prof = hqt.seed.stationary_profile(6.0, -2 * np.pi * 7 / 20)
    state = list(hqt.seed.init_driven(nx, ny, nz, prof, noise="complex", amplitude=1e-2, seed=3))
    state[0] = state[0] * np.exp(2j * np.pi * np.arange(ny) / ny)[None, :, None]
    op = oracle.build_operators(nx, ny, nz, L)
    want, w = oracle.rk4_step(op, oracle.OracleState(*[a.copy() for a in state]), 0.005, 6.0,
                              prof.vy, True)
    with hqt.Simulation(nx, ny, nz, Lx=L, Ly=L, mu=6.0, vy=prof.vy, dt=0.005) as sim:
        got, info = sim.step(*state, nsteps=1)
        O = oracle.boundary_order_parameter(op, vortex_field(nx, ny, nz, 2, seed=nx))
        k, E, _, _ = oracle.energy_spectrum(O, L, L)
        gk, gE, _, _ = sim.energy_spectrum_device(to_d(O[:, :, None])[0])
    assert info.last_winding == w
    for g, r in zip(got, (want.Z1, want.Z2, want.Z3, want.Z4, want.rhoi)):
        assert np.linalg.norm((g - r).ravel()) < 1e-12 * max(np.linalg.norm(r.ravel()),
                                                             np.linalg.norm(want.Z2.ravel()))
    assert np.allclose(gk, k, rtol=1e-14)
    # a mode on a shell edge may be binned on either side of it: the cumulative
    # sum differs by no more than one shell there
    assert abs(gE.sum() - E.sum()) < 1e-9 * E.sum()
