"""d/dy in the FP64 path's inverse Chebyshev transforms (csrc/cheb_oz.cu) against extended precision.

The field is the (0,0) mode alone, u = (U, V, W)(y): N(u) holds products of U, V, W and their derivatives and nothing of
the x and z transforms' wavenumbers.  Tolerance: the derivative's terms n^2 x_n, the products and the forward transform
are each rounded to a few eps of values no larger than the largest of their sums; 16 eps of the norm of N(u) bounds them
(products in double precision: 1 to 3 eps).  Coefficients rounded before their weights 2n would be off by up to
N^2 2^-61 of the sum of n^2 |x_n|: 30 eps at Ny = 49, 600 at 139.
"""

import numpy as np
import pytest

from oracle import cf_oracle as O
from tests.helpers import COUETTE_BOX, to_cflags, to_cgrid

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps
PI = np.longdouble("3.14159265358979323846264338327950288")


@pytest.fixture(scope="module", autouse=True)
def built():
    from channelflow_gb300 import build
    build.build()


def _matrices(N):
    """Inverse transform, its derivative (y in [-1, 1]) and forward transform in extended precision."""
    j = np.arange(N)
    m = np.outer(j, j) % (2 * (N - 1))
    T = np.cos(PI * m.astype(np.longdouble) / np.longdouble(N - 1))
    D = np.sin(PI * m.astype(np.longdouble) / np.longdouble(N - 1)) * j
    D[1:-1] /= np.sin(PI * j[1:-1].astype(np.longdouble) / np.longdouble(N - 1))[:, None]
    D[0] = j.astype(np.longdouble) ** 2
    D[-1] = np.where(j % 2, 1, -1) * j.astype(np.longdouble) ** 2
    e = np.where((j == 0) | (j == N - 1), np.longdouble(0.5), np.longdouble(1))
    return T, D, T * np.outer(e, e) * 2 / np.longdouble(N - 1)


# both kernels of few and of many lines, around the K steps of 16 and the largest covered lengths
@pytest.mark.parametrize("dims", [(6, 17, 6), (6, 33, 6), (6, 49, 6), (64, 49, 64), (64, 63, 64), (6, 63, 6), (6, 65, 6),
                                  (6, 97, 6), (6, 111, 6), (6, 129, 6), (6, 139, 6)], ids=str)
@pytest.mark.parametrize("form", [O.Rotational, O.Convection])
@pytest.mark.parametrize("decay", [0.6, 0.95, 1.0])
def test_mean_profile(dims, form, decay):
    from channelflow_gb300 import DNS
    if dims[1] > 111 and form != O.Rotational:
        pytest.skip("Ny > 111 takes the rotational form only")
    g = O.Grid(*dims, *COUETTE_BOX)
    N = g.Ny
    fl = O.DNSFlags(nu=1 / 400, dt=0.02, baseflow=O.ZeroBase, nonlinearity=form)
    rng = np.random.default_rng(N)
    x = rng.standard_normal((3, N)) * decay ** np.arange(N)
    u = np.zeros((3, N, g.Nx, g.Mz), complex)
    u[:, :, 0, 0] = x
    d = DNS(np.zeros_like(u), to_cgrid(g), to_cflags(fl))
    got = d.nonlinear(u)[:, :, 0, 0]
    d.close()
    T, D, F = _matrices(N)
    x = x.astype(np.longdouble)
    U, V, W = (T @ c for c in x)
    dU, dV, dW = (D @ c for c in x)
    if form == O.Rotational:  # vorticity (W', 0, -U') x (U, V, W)
        ref = [dU * V, -dU * U - dW * W, dW * V]
    else:
        ref = [V * dU, V * dV, V * dW]
    ref = np.array([F @ r for r in ref])
    assert np.linalg.norm((got.real - ref).astype(float)) <= 16 * EPS * np.linalg.norm(ref.astype(float))
