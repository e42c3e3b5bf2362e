"""FP64 transforms and nonlinear terms of single waves and point impulses: lines with one non-zero element.

Tolerance of a transform: 32 eps of the plane's sum of magnitudes (two FFTs of at most 9 stages on each side).  Nonlinear
terms: 1000 eps, as for dense spectra at these Ny (Chebyshev derivatives of 9 points).
"""

import numpy as np
import pytest

from oracle import cf_oracle as O
from tests.helpers import COUETTE_BOX, rel_l2, to_cflags, to_cgrid

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps
LENGTHS = [16, 32, 48, 64, 96, 128, 256, 320, 384, 448, 512]


@pytest.fixture(scope="module", autouse=True)
def built():
    from channelflow_gb300 import build
    build.build()


def _amplitudes(n, seed):
    """Real, imaginary and random phases in turn, moduli from 1 to 2."""
    rng = np.random.default_rng(seed)
    phase = np.exp(2j * np.pi * rng.random(n))
    phase[0::3], phase[1::3] = 1.0, 1j
    return phase * rng.uniform(1, 2, n)


@pytest.mark.parametrize("L", LENGTHS)
@pytest.mark.parametrize("along", ["x", "z"])
def test_transforms(along, L):
    """One mode a plane to physical, one point a plane to spectral, at every index of the long direction."""
    from channelflow_gb300.flowfield import FlowField, Physical
    Nx, Nz = (L, 6) if along == "x" else (6, L)
    Mz, planes = Nz // 2 + 1, 2 * L
    i = np.arange(planes)
    amp = _amplitudes(planes, L)
    f = FlowField(Nx, 2, Nz, planes // 2, 2.0, 1.0)
    u = np.zeros((planes, Nx, Mz), complex)
    u[i, i % Nx, i % Mz] = amp
    f.set_raw(u.view(float).reshape(planes // 2, 2, Nx, 2 * Mz), 1, Physical)
    f.makePhysical_xz()
    ref = np.fft.irfft(np.fft.ifft(u, axis=1) * Nx, n=Nz, axis=2) * Nz
    got = f.physical().reshape(planes, Nx, Nz)
    assert np.all(np.abs(got - ref) <= 32 * EPS * 2 * np.abs(amp)[:, None, None])
    p = np.zeros((planes, Nx, Nz))
    p[i, i % Nx, i % Nz] = amp.real + amp.imag
    f.set_physical(p.reshape(planes // 2, 2, Nx, Nz))
    f.makeSpectral_xz()
    got = f.spectral().reshape(planes, Nx, Mz) * (Nx * Nz)
    ref = np.fft.rfft2(p, axes=(1, 2))
    assert np.all(np.abs(got - ref) <= 32 * EPS * np.abs(p).sum((1, 2))[:, None, None])


@pytest.mark.parametrize("form", [O.Rotational, O.SkewSymmetric])
@pytest.mark.parametrize("dims", [(64, 9, 12), (256, 9, 12), (320, 9, 12), (12, 9, 64), (12, 9, 320), (96, 9, 96)], ids=str)
def test_oblique_wave(dims, form):
    """N(u) of one oblique wave on a laminar base flow, for several of the solved modes."""
    from channelflow_gb300 import DNS
    g = O.Grid(*dims, *COUETTE_BOX)
    fl = O.DNSFlags(nu=1 / 400, dt=0.02, baseflow=O.LaminarBase, ulowerwall=-1.0, uupperwall=1.0, nonlinearity=form)
    rng = np.random.default_rng(sum(dims))
    d = DNS(np.zeros((3, g.Ny, g.Nx, g.Mz), complex), to_cgrid(g), to_cflags(fl))
    kxm, kzm = g.Nx // 3 - 1, g.Nz // 3 - 1
    for kx, kz in {(1, 1), (kxm, 1), (min(5, kxm), kzm), (-1, kzm), (-min(3, kxm), min(2, kzm))}:
        u = np.zeros((3, g.Ny, g.Nx, g.Mz), complex)
        u[:, :, kx, kz] = _amplitudes(3 * g.Ny, kx + 100 * kz).reshape(3, g.Ny) * 0.7 ** np.arange(g.Ny)
        u[:, :, kx, kz] *= rng.uniform(1, 2)
        ref, _ = O.NSE(g, fl, None, u).nonlinear(u.copy())
        assert rel_l2(d.nonlinear(u), ref, g) <= 1000 * EPS
    d.close()
