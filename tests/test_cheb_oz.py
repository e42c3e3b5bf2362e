"""FP64 Chebyshev transforms by exact integer products on the tensor cores (csrc/cheb_oz.cu).

Tolerances.  One transform: input and output rounding and the matrix's 62 bits are below 2 eps of the line's sum of
magnitudes, the reference (extended precision where the host has it) below N eps of it.  Nonlinear terms: the oracle's
FFTs and Chebyshev sums carry a few eps per stage, which a derivative amplifies by up to N on average: 100 N eps.
"""

import numpy as np
import pytest

from oracle import cf_oracle as O
from tests.helpers import COUETTE_BOX, rel_l2, to_cflags, to_cgrid

EPS = np.finfo(float).eps
# around the K steps of 16 points and the units of 8 rows per parity, the largest covered lengths, one beyond
NY = [3, 4, 5, 15, 16, 17, 31, 32, 33, 35, 47, 49, 63, 65, 95, 97, 111, 127, 129, 139, 145]


@pytest.fixture(scope="module", autouse=True)
def built():
    from channelflow_gb300 import build
    build.build()


def _cos(N):
    j = np.arange(N)
    pi = np.longdouble("3.14159265358979323846264338327950288")
    return np.cos(pi * (np.outer(j, j) % (2 * (N - 1))).astype(np.longdouble) / np.longdouble(N - 1))


@pytest.mark.gpu
@pytest.mark.parametrize("Ny", NY)
def test_y_transforms(Ny):
    """Both directions, dense and decaying spectra, line scales from 2^-300 to 2^300, 133 x 2 lines (ragged tile)."""
    from channelflow_gb300.flowfield import FlowField, Physical, Spectral
    Nx, Nz, Nd = 14, 36, 7
    rng = np.random.default_rng(Ny)
    x = rng.standard_normal((Nd, Ny, Nx, Nz + 2))
    x[1] *= (0.6 ** np.arange(Ny))[:, None, None]
    x[2] = np.ldexp(x[2], rng.integers(-300, 300, (1, Nx, Nz + 2)))
    x[3, :, 2:5] = 0
    T = _cos(Ny)
    e = np.where((np.arange(Ny) == 0) | (np.arange(Ny) == Ny - 1), 0.5, 1.0)
    F = T * np.outer(e, e) * 2 / np.longdouble(Ny - 1)
    f = FlowField(Nx, Ny, Nz, Nd, 2.0, 1.0)
    mag = np.abs(x).sum(1, keepdims=True)
    for M, state, go in ((T, Spectral, "makePhysical_y"), (F, Physical, "makeSpectral_y")):
        f.set_raw(x, Spectral, state)
        getattr(f, go)()
        got = f.raw().reshape(x.shape)
        ref = np.einsum("jn,cnxz->cjxz", M, x.astype(np.longdouble)).astype(float)
        assert np.all(np.abs(got - ref) <= (4 + Ny) * EPS * mag)
    x[4, 1, 3, 5], x[5, 2, 4, 6] = np.nan, -np.inf
    f.set_raw(x, Spectral, Spectral)
    f.makePhysical_y()
    got = f.raw().reshape(x.shape)
    bad = np.zeros(x.shape, bool)
    bad[4, :, 3, 5] = bad[5, :, 4, 6] = True
    assert np.all(np.isnan(got[4, :, 3, 5])) and not np.any(np.isfinite(got[5, :, 4, 6]))
    assert np.all(np.isfinite(got[~bad]))


def _random(g, seed):
    rng = np.random.default_rng(seed)
    u = rng.standard_normal((3, g.Ny, g.Nx, g.Nz))
    s = np.fft.rfft2(u, axes=(2, 3)) * (0.7 ** np.arange(g.Ny))[None, :, None, None]
    return np.ascontiguousarray(s / (g.Nx * g.Nz))


@pytest.mark.gpu
@pytest.mark.parametrize("form", [O.Rotational, O.Convection, O.Divergence, O.SkewSymmetric])
@pytest.mark.parametrize("Ny", [5, 15, 17, 33, 47, 65, 97, 111])
def test_nonlinear_matches_oracle(Ny, form):
    """Base flow, suction and a domain of length 3/2; the curl with the fused x/z pass too."""
    from channelflow_gb300 import DNS
    from channelflow_gb300 import _lib as L
    g = O.Grid(32, Ny, 48, *COUETTE_BOX, a=-0.5, b=1.0)
    fl = O.DNSFlags(nu=1 / 400, dt=0.02, baseflow=O.LaminarBase, ulowerwall=-1.0, uupperwall=1.0, Vsuck=0.02,
                    nonlinearity=form)
    u = O.zero_padded_modes(_random(g, Ny), g)
    ref, _ = O.NSE(g, fl, None, u).nonlinear(u.copy())
    for fused in (0, 2) if form == O.Rotational else (0,):
        L.check(L.load().cfgpu_set_fused_xz(fused))
        try:
            d = DNS(u.copy(), to_cgrid(g), to_cflags(fl))
            f = d.nonlinear(u)
            d.close()
        finally:
            L.check(L.load().cfgpu_set_fused_xz(1))
        assert rel_l2(f, ref, g) <= 100 * Ny * EPS


@pytest.mark.gpu
@pytest.mark.parametrize("Ny", [3, 16, 17, 33, 34, 49, 63, 64])
def test_few_lines_same_bits(Ny):
    """One component (CTAs of 32 lines) and the same one among seven (CTAs of 128): exact products, equal results."""
    from channelflow_gb300.flowfield import FlowField, Physical, Spectral
    Nx, Nz = 30, 36
    x = np.random.default_rng(Ny).standard_normal((7, Ny, Nx, Nz + 2)) * (0.8 ** np.arange(Ny))[None, :, None, None]
    x[0, :, 3, 4] = 0
    x[0, Ny // 2, 5, 6] = np.nan
    for state, go in ((Spectral, "makePhysical_y"), (Physical, "makeSpectral_y")):
        got = []
        for Nd in (7, 1):
            f = FlowField(Nx, Ny, Nz, Nd, 2.0, 1.0)
            f.set_raw(np.ascontiguousarray(x[:Nd]), Spectral, state)
            getattr(f, go)()
            got.append(f.raw().reshape(x[:Nd].shape)[0])
        assert np.array_equal(got[0], got[1], equal_nan=True)
