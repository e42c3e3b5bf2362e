"""A wait that runs out in a tensor-core transform reaches the caller: the flag that such a kernel sets is set from the
host here (no kernel is disturbed), and every call that waits for results returns CFGPU_ECUDA with a message."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
GRID = (16, 17, 16)


@pytest.fixture(scope="module", autouse=True)
def built():
    from channelflow_gb300 import build
    build.build()


def _field(seed=1):
    from channelflow_gb300.fields import random_divfree_field
    return random_divfree_field(*GRID, 2.0, 1.0, seed=seed, norm=0.1)


def _raises(f):
    from channelflow_gb300 import _lib as L
    with pytest.raises(L.CfgpuError, match="wait"):
        f()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_dns(precision):
    from channelflow_gb300 import DNS, DNSFlags, Grid
    from channelflow_gb300 import _lib as L
    u = _field()
    q = np.zeros((1,) + u.shape[1:], complex)
    d = DNS(u.copy(), Grid(*GRID, 2.0, 1.0), DNSFlags(nu=0.01, dt=0.01), precision=precision)
    other = DNS(u.copy(), Grid(*GRID, 2.0, 1.0), DNSFlags(nu=0.01, dt=0.01), precision=precision)
    d.advance(u, q, 3)
    lib = L.load()
    L.check(lib.cfgpu_dns_inject_wait_error(d._h))
    x = C.c_double()
    f = np.empty_like(u)
    for call in (lambda: d.advance(u, q, 1), lambda: d.nonlinear(u),
                 lambda: L.check(lib.cfgpu_dns_cfl(d._h, C.byref(x))),
                 lambda: L.check(lib.cfgpu_dns_l2norm(d._h, 0, C.byref(x))),
                 lambda: L.check(lib.cfgpu_dns_advance_resident(d._h, 1)),
                 lambda: L.check(lib.cfgpu_dns_advance_timed(d._h, 1, C.byref(x))),
                 lambda: L.check(lib.cfgpu_dns_get_fields(d._h, L.dptr(f.view(float)), None))):
        _raises(call)
    other.advance(u, q, 3)  # another object is not concerned
    d.close()
    other.close()
    d = DNS(u.copy(), Grid(*GRID, 2.0, 1.0), DNSFlags(nu=0.01, dt=0.01), precision=precision)  # the flag's memory again
    d.advance(u, q, 1)
    d.close()


def test_ensemble():
    from channelflow_gb300 import DNSFlags, Ensemble, Grid
    from channelflow_gb300 import _lib as L
    e = Ensemble(Grid(*GRID, 2.0, 1.0), DNSFlags(nu=0.01, dt=0.01), 2)
    u = _field()
    q = np.zeros((1,) + u.shape[1:], complex)
    for s in range(2):
        e.set_field(s, _field(s + 1))
    e.advance_resident(2)
    e.get_field(1, u, q)
    L.check(L.load().cfgpu_dns_inject_wait_error(e._h))
    _raises(lambda: e.get_field(1, u, q))
    _raises(e.dPdx)
    _raises(e.CFL)
    e.close()


def test_flowfield():
    from channelflow_gb300 import _lib as L
    from channelflow_gb300.flowfield import FlowField
    u = _field()
    f = FlowField(*GRID, 3, 2.0, 1.0)
    f.set_spectral(u)
    f.makePhysical()
    ref = f.physical()
    L.check(L.load().cfgpu_flowfield_inject_wait_error(f._h))
    _raises(f.makeSpectral)
    _raises(f.raw)
    f.set_spectral(u)  # new data
    f.makePhysical()
    assert np.array_equal(f.physical(), ref)
    assert L.load().cfgpu_dns_inject_wait_error(None) == L.CFGPU_EINVAL
    assert L.load().cfgpu_flowfield_inject_wait_error(None) == L.CFGPU_EINVAL
