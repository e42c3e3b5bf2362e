"""The FP64 path's x/z passes on 64-bit integers (csrc/fx.cuh, csrc/xz_fx.cu) against the oracle's nonlinear term.

Tolerance: the transforms of both sides carry a few rounding units per stage; 1000 of them (2.2e-13 relative L2)
bound the longest chain here with the Chebyshev derivatives of Ny <= 17 points.
"""

import numpy as np
import pytest

from oracle import cf_oracle as O
from tests.helpers import COUETTE_BOX, rel_l2, to_cflags, to_cgrid

TOL = 1000 * np.finfo(float).eps
# lengths around the compile-time ones, every radix (2, 3, 4, 5, 7, 11, 13), single solved wavenumbers, row counts
# that leave the last block of the z pass ragged
GRIDS = [(4, 9, 6), (6, 9, 4), (10, 9, 32), (30, 9, 22), (34, 9, 26), (50, 9, 28), (64, 17, 96), (128, 9, 10), (14, 9, 128),
         (160, 9, 48),
         # radices 6, 8, 9, 10, 12, 15, 16, single stages, three stages, a prime behind a composite
         (144, 9, 8), (8, 9, 192), (90, 9, 72), (36, 9, 150), (256, 9, 12), (16, 9, 270), (224, 9, 14)]


@pytest.fixture(autouse=True)
def three_kernel_path():
    """The x and z passes as separate kernels (small grids would otherwise take the fused FP64 kernel)."""
    from channelflow_gb300 import _lib as L
    from channelflow_gb300 import build
    build.build()
    L.check(L.load().cfgpu_set_fused_xz(0))
    yield
    L.check(L.load().cfgpu_set_fused_xz(1))


def _random(g, decay, seed):
    rng = np.random.default_rng(seed)
    u = rng.standard_normal((3, g.Ny, g.Nx, g.Nz))
    s = np.fft.rfft2(u, axes=(2, 3)) * (0.7 ** np.arange(g.Ny))[None, :, None, None]
    k = np.abs(np.fft.fftfreq(g.Nx, 1 / g.Nx))[:, None] + np.arange(g.Mz)[None, :]
    return np.ascontiguousarray(s * decay ** k / (g.Nx * g.Nz))


def _nonlinear(u, g, fl):
    from channelflow_gb300 import DNS
    d = DNS(u.copy(), to_cgrid(g), to_cflags(fl))
    f = d.nonlinear(u)
    d.close()
    return f


@pytest.mark.gpu
@pytest.mark.parametrize("form", [O.Rotational, O.Convection, O.Divergence, O.SkewSymmetric])
@pytest.mark.parametrize("dims", GRIDS, ids=str)
def test_matches_oracle(dims, form):
    g = O.Grid(*dims, *COUETTE_BOX)
    fl = O.DNSFlags(nu=1 / 400, dt=0.02, baseflow=O.LaminarBase, ulowerwall=-1.0, uupperwall=1.0, nonlinearity=form)
    u = O.zero_padded_modes(_random(g, 0.8, 5), g)
    ref, _ = O.NSE(g, fl, None, u).nonlinear(u.copy())
    assert rel_l2(_nonlinear(u, g, fl), ref, g) <= TOL


@pytest.mark.gpu
def test_without_dealiasing():
    g = O.Grid(16, 9, 18, *COUETTE_BOX)
    fl = O.DNSFlags(nu=1 / 400, dt=0.02, baseflow=O.ZeroBase, dealiasing=O.NoDealiasing)
    u = _random(g, 0.8, 6)
    u[:, :, g.Nx // 2] = 0
    u[:, :, :, g.Nz // 2] = 0
    ref, _ = O.NSE(g, fl, None, u).nonlinear(u.copy())
    ref[:, :, g.Nx // 2] = 0
    ref[:, :, :, g.Nz // 2] = 0
    assert rel_l2(_nonlinear(u, g, fl), ref, g) <= TOL


@pytest.mark.gpu
@pytest.mark.parametrize("form", [O.Rotational, O.SkewSymmetric])
def test_scale_zero_and_nonfinite(form):
    """Lines are scaled by powers of two: N(2^s u) = 2^2s N(u) bit for bit; zero fields and components give zeros; a
    line with an infinite or NaN coefficient gives NaN, other planes nothing."""
    g = O.Grid(20, 9, 24, *COUETTE_BOX)
    fl = O.DNSFlags(nu=1 / 400, dt=0.02, baseflow=O.ZeroBase, nonlinearity=form)
    u = O.zero_padded_modes(_random(g, 0.8, 7), g)
    f = _nonlinear(u, g, fl)
    for s in (-450, 450):
        assert np.array_equal(_nonlinear(np.ldexp(u.view(float), s).view(complex), g, fl).view(float),
                              np.ldexp(f.view(float), 2 * s))
    assert not np.any(_nonlinear(np.zeros_like(u), g, fl))
    w = u.copy()
    w[1:] = 0  # only u: one velocity component is zero at every point
    ref, _ = O.NSE(g, fl, None, w).nonlinear(w.copy())
    assert rel_l2(_nonlinear(w, g, fl), ref, g) <= TOL
    for bad in (np.nan, np.inf):
        w = u.copy()
        w[0, 2, 1, 3] = bad
        assert np.all(np.isnan(_nonlinear(w, g, fl)[:, :, :5, :7].real))
