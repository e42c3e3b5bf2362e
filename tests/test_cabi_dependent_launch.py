"""Programmatic dependent launch (cfgpu_set_pdl) on and off: the same bits.

With it a kernel is scheduled while its predecessor still runs and waits for that kernel's results itself
(common.cuh): a wait in the wrong place would show as a difference.  Off, the default, is left behind.
"""

import numpy as np
import pytest

from channelflow_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def default_launches():
    from channelflow_gb300 import build
    build.build()
    yield
    L.check(L.load().cfgpu_set_pdl(0))


def _advance(grid, flags, u0, precision, pdl):
    from channelflow_gb300 import DNS
    L.check(L.load().cfgpu_set_pdl(pdl))
    u = u0.copy()
    q = np.zeros((1,) + u.shape[1:], complex)
    d = DNS(u, grid, flags, precision=precision)
    n = d.nonlinear(u)
    for steps in (3, 6):  # start-up and captured steps
        d.advance(u, q, steps)
    d.close()
    return n, u, q


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("form", ["Rotational", "SkewSymmetric", "Convection"])
@pytest.mark.parametrize("scheme", ["SBDF3", "CNAB2", "SMRK2"])
@pytest.mark.parametrize("dims", [(24, 33, 24), (40, 49, 36), (48, 65, 48)], ids=str)
def test_same_bits(dims, scheme, form, precision):
    from channelflow_gb300 import DNSFlags, Grid
    from channelflow_gb300 import dns as D
    from channelflow_gb300.fields import random_divfree_field
    g = Grid(*dims, 5.5, 2.5)
    fl = DNSFlags(nu=1 / 400, dt=0.01, baseflow=D.LaminarBase, ulowerwall=-1.0, uupperwall=1.0,
                  timestepping=getattr(D, scheme), nonlinearity=getattr(D, form))
    u0 = np.ascontiguousarray(random_divfree_field(*dims, 5.5, 2.5, seed=3, norm=0.2))
    off = _advance(g, fl, u0, precision, 0)
    for _ in range(2):
        for a, b in zip(off, _advance(g, fl, u0, precision, 1)):
            assert np.array_equal(a, b)
