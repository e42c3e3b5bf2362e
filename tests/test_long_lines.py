"""FP64 x and z transforms of long lines: no less exact than double-precision FFTs.

Flat data: the relative rms error of a double-precision FFT of length L is about eps sqrt(log2 L) / 3 (radix 4: 0.3 to
0.35 of eps sqrt(log2 L)), and 0.6 eps sqrt(log2 L) allows for the short transform of the other direction and the rounding
of the input.  Fixed-point lines scaled by their sum of magnitudes lose sqrt(L) against that.
"""

import numpy as np
import pytest

from oracle import cf_oracle as O
from tests.helpers import COUETTE_BOX, rel_l2, to_cflags, to_cgrid

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


@pytest.fixture(scope="module", autouse=True)
def built():
    from channelflow_gb300 import build
    build.build()


def _rel(a, b):
    return float(np.sqrt(np.sum(np.abs(a - b) ** 2) / np.sum(np.abs(b) ** 2)))


@pytest.mark.parametrize("L", [320, 336, 338, 360, 384, 512, 640, 1024, 1500, 2048, 2916, 3000])
@pytest.mark.parametrize("along", ["x", "z"])
def test_flat_fields(along, L):
    from channelflow_gb300.flowfield import FlowField, Physical, Spectral
    Nx, Nz = (L, 6) if along == "x" else (6, L)
    Mz = Nz // 2 + 1
    rng = np.random.default_rng(L)
    tol = 0.6 * EPS * np.sqrt(np.log2(L))
    f = FlowField(Nx, 2, Nz, 2, 2.0, 1.0)
    p = rng.standard_normal((2, 2, Nx, Nz))
    f.set_physical(p)
    f.makeSpectral_xz()
    q = p.astype(np.longdouble)
    ref = np.fft.fft(np.fft.rfft(q, axis=3), axis=2) / (Nx * Nz)
    assert _rel(f.spectral(), ref) <= tol
    u = rng.standard_normal((2, 2, Nx, Mz)) + 1j * rng.standard_normal((2, 2, Nx, Mz))
    f.set_raw(u.view(float), Spectral, Physical)
    f.makePhysical_xz()
    ref = np.fft.irfft(np.fft.ifft(u.astype(np.clongdouble), axis=2) * Nx, n=Nz, axis=3) * Nz
    assert _rel(f.physical(), ref) <= tol


@pytest.mark.parametrize("form", [O.Rotational, O.Convection, O.Divergence, O.SkewSymmetric])
@pytest.mark.parametrize("dims", [(336, 9, 8), (360, 9, 8), (640, 9, 6), (6, 9, 336), (6, 9, 360), (8, 9, 594), (384, 9, 384)],
                         ids=str)
def test_nonlinear(dims, form):
    """Around the line lengths where the FP64 DNS passes change their arithmetic, x and z apart and together."""
    from channelflow_gb300 import DNS
    g = O.Grid(*dims, *COUETTE_BOX)
    fl = O.DNSFlags(nu=1 / 400, dt=0.02, baseflow=O.LaminarBase, ulowerwall=-1.0, uupperwall=1.0, nonlinearity=form)
    rng = np.random.default_rng(sum(dims))
    s = np.fft.rfft2(rng.standard_normal((3, g.Ny, g.Nx, g.Nz)), axes=(2, 3)) * (0.7 ** np.arange(g.Ny))[None, :, None, None]
    u = O.zero_padded_modes(np.ascontiguousarray(s / (g.Nx * g.Nz)), g)
    d = DNS(u.copy(), to_cgrid(g), to_cflags(fl))
    ref, _ = O.NSE(g, fl, None, u).nonlinear(u.copy())
    assert rel_l2(d.nonlinear(u), ref, g) <= 1000 * EPS
    d.close()
