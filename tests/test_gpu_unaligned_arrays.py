"""Host arrays that do not start on an 8-byte boundary (views into packed
records): every call that takes or fills a field gives the values that aligned
arrays give."""
import numpy as np
import pytest

from nextsimdg_gb300.dynamics import MEVPDynamicsKernel
from nextsimdg_gb300.ice_growth import IceGrowth
from test_gpu_step_preparation import _fields
from test_stress_metric import _coords

pytestmark = pytest.mark.gpu


def _odd(a, offset=1):
    """The values of a at an address offset bytes past an 8-byte boundary."""
    b = np.empty(a.nbytes + 16, dtype=np.uint8)
    start = -b.ctypes.data % 8 + offset
    v = b[start:start + a.nbytes].view(np.float64)
    v[:] = a.ravel()
    assert v.ctypes.data % 8 == offset
    return v


@pytest.mark.parametrize("offset", [1, 4])
def test_dynamics(gpu, offset):
    nx, ny = 31, 17
    f = _fields(nx, ny, False)
    got = []
    for odd in (False, True):
        k = MEVPDynamicsKernel(dg_comp=3, n_steps=5)
        k.initialise(_coords("box", nx, ny), False, np.ones((ny, nx)))
        take = (lambda a: _odd(a, offset)) if odd else (lambda a: a)
        for name, a in f.items():
            k.setData(name, take(a))
        out = {name: take(np.zeros(nx * ny)) for name in ("u", "v", "hice", "uiostress")}
        k.module_step(0.0, 120.0, {name: take(f[name]) for name in ("hice", "uwind", "vwind", "ssh")}, out)
        u = take(np.zeros(nx * ny))
        k.getDG0Data("v", u)
        got.append([*out.values(), u])
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("n", [100, 30000])
def test_growth(gpu, n):
    rng = np.random.default_rng(2)
    g = IceGrowth(n)
    for name in ("hice", "cice"):
        a = rng.uniform(0.1, 1.0, n)
        g.setData(name, _odd(a))
        np.testing.assert_array_equal(g.getData(name), a)
        out = _odd(np.zeros(n))
        g._check(g._l.nsdg_ice_growth_get_field(g._h, name.encode(), out.ctypes.data, n))
        np.testing.assert_array_equal(out, a)
