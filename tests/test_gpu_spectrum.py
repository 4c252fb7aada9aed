"""The energy spectrum, shell by shell, of a field with energy in every mode: a row of the
y transform out of place moves energy between shells.  Runtime plans along y of two,
three and four passes, compile-time ones, and the prime-factor engine along x.  With
(Ly/Lx)^2 irrational no mode but those of one axis, whose wavenumber both sides form alike,
lies near a shell's edge."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(64, 96), (50, 180), (96, 250), (301, 40), (36, 750),
                                   (250, 64), (40, 1024), (48, 1500), (31, 37)])
def test_every_shell(hqt, oracle, dev, nx, ny):
    to_d, _ = dev
    Lx, Ly = 0.4 * nx, 0.4 * np.pi / 3 * ny
    rng = np.random.default_rng(nx + ny)
    O = 1.0 + 0.2 * (rng.standard_normal((nx, ny)) + 1j * rng.standard_normal((nx, ny)))
    k, E, Ec, Ei = oracle.energy_spectrum(O, Lx, Ly)
    with hqt.Simulation(nx, ny, 5, Lx=Lx, Ly=Ly) as sim:
        gk, gE, gEc, gEi = sim.energy_spectrum_device(to_d(O[:, :, None])[0])
    assert len(gk) == len(k) and np.allclose(gk, k, rtol=1e-14)
    for got, want in ((gE, E), (gEc, Ec), (gEi, Ei)):
        assert np.max(np.abs(got - want)) < 1e-9 * E.max()
