"""The plain sub-cycle inside a warm-started step (the fallback, an audit)
starts from the restored velocity and divergence: bitwise the plain update, on
each of the mixed path's element kernels, one thread per element or three."""
import numpy as np
import pytest

from nextsimdg_gb300 import surrogate
from nextsimdg_gb300.dynamics import MEVPDynamicsKernel
from test_gpu_step_preparation import _fields
from test_stress_metric import _coords

pytestmark = pytest.mark.gpu

K, STEPS, DT = 12, 6, 120.0


def _kernel(kind, nx, ny):
    k = MEVPDynamicsKernel(dg_comp=3, n_steps=30, precision=1)
    k.initialise(_coords(kind, nx, ny), kind == "sphere", np.ones((ny, nx)))
    for name, a in _fields(nx, ny, False).items():
        k.setData(name, a)
    return k


@pytest.mark.parametrize("kind", ["sheared", "quads", "sphere"])
@pytest.mark.parametrize("nx,ny", [(40, 24), (160, 112)])
@pytest.mark.parametrize("audit", [0, 1])
def test_bitwise_the_plain_update(gpu, kind, nx, ny, audit):
    net = surrogate.warm_net(nx, ny)
    net.dataset_reserve(2)
    sampled = _kernel(kind, nx, ny)
    for s in range(2):
        sampled.warm_sample(s * DT, DT, K, net, s)
    net.dataset_normalise(2)
    plain, warm = _kernel(kind, nx, ny), _kernel(kind, nx, ny)
    warm.set_warm_start(net, K, 0.0, audit_every=audit, audit_tol=1e9)  # every step falls back, or is audited
    for s in range(STEPS):
        plain.update(s * DT, DT)
        warm.update(s * DT, DT)
        for name in ("u", "v", "hice", "cice"):
            np.testing.assert_array_equal(plain.getDG0Data(name), warm.getDG0Data(name), err_msg=f"{name}, step {s}")
    st = warm.warm_stats()
    assert (st["audited"], st["fallbacks"]) == ((STEPS, 0) if audit else (0, STEPS))
